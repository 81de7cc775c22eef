// FRI folds over QM31, and the commit phase's small layers.
//
// fri.zig:209-219 folds y0 = L[j], y1 = L[j + n/2] at x = D_i[j] into
//   (y0 + y1) * inv2 + alpha * ((y0 - y1) * x^-1 * inv2).
// x^-1 is rebuilt from tables instead of a per-point inversion: D_i[j] is a unit of
// the QM31 ring, so its inverse is unique and equals
// (FRI_OFFSET^(2^i))^-1 * w_0^-(j * 2^i), w_0 = primitiveRootOfUnity(dlog). inv2 = 2^30.
#include "blake3.cuh"
#include "fri.cuh"
#include "host.cuh"
#include "transcript.cuh"
#include "tree.cuh"

namespace zs {

__global__ void k_fold_tables(qm31 w0inv, qm31* tabs) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= 3 * 2048) return;
  const uint32_t which = k / 2048, e = k % 2048;
  // w0inv^(e * 2^(11 * which))
  qm31 base = w0inv;
  for (uint32_t s = 0; s < 11 * which; ++s) base = qmul(base, base);
  tabs[k] = qpow(base, e);
}

FoldTables::FoldTables(unsigned d, cudaStream_t s) : dlog(d), st(s) {
  if (dlog > 32) throw Error(ZS_EMALFORMED, "FRI domain log size above 32");
  ZS_CUDA(cudaMallocAsync(&tables, 3 * 2048 * sizeof(qm31), st));
  const qm31 w0 = q_root_of_unity(dlog);
  k_fold_tables<<<(3 * 2048 + 255) / 256, 256, 0, st>>>(qinv(w0), tables);
  ZS_CUDA(cudaGetLastError());
}
FoldTables::~FoldTables() { cudaFreeAsync(tables, st); }

qm31 FoldTables::offset_inv(unsigned layer) const { return qinv(qpow(q_fri_offset(), (uint64_t)1 << layer)); }

namespace {
constexpr unsigned kThreads = 256;
}  // namespace

// One fold output per thread.
__global__ void __launch_bounds__(kThreads) k_fold(const qm31* __restrict__ in, qm31* __restrict__ out, uint32_t half,
                                                   qm31 alpha, const qm31* __restrict__ alpha_dev, qm31 off_inv,
                                                   unsigned layer, const qm31* __restrict__ tabs) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= half) return;
  const uint4* src = reinterpret_cast<const uint4*>(in);
  if (alpha_dev) alpha = q_of(__ldg(reinterpret_cast<const uint4*>(alpha_dev)));
  reinterpret_cast<uint4*>(out)[j] =
      u4_of(fold_value(q_of(__ldg(src + j)), q_of(__ldg(src + j + half)), j, layer, qmul(alpha, off_inv), tabs));
}

void fri_fold(const qm31* d_in, qm31* d_out, uint32_t half, const qm31& alpha, const qm31* d_alpha, unsigned layer,
              const FoldTables& tabs, cudaStream_t st) {
  k_fold<<<(half + kThreads - 1) / kThreads, kThreads, 0, st>>>(d_in, d_out, half, alpha, d_alpha,
                                                                tabs.offset_inv(layer), layer, tabs.tables);
  ZS_CUDA(cudaGetLastError());
}

constexpr unsigned kChainThreads = 512;
__global__ void __launch_bounds__(kChainThreads) k_fold_chain(const __grid_constant__ FoldChain fc) {
#pragma unroll 1
  for (unsigned i = 0; i < fc.count; ++i) {
    const uint32_t half = 1u << (fc.log_size - i - 1);
    const uint4* in = reinterpret_cast<const uint4*>(fc.layer[i]);
    uint4* out = reinterpret_cast<uint4*>(fc.layer[i + 1]);
    for (uint32_t j = threadIdx.x; j < half; j += blockDim.x)
      out[j] = u4_of(fold_value(q_of(__ldcg(in + j)), q_of(__ldcg(in + j + half)), j, fc.first + i, fc.c[i], fc.tables));
    __syncthreads();
  }
}

void fri_fold_chain(const FoldChain& chain, cudaStream_t st) {
  if (chain.count == 0) return;
  if (chain.log_size > kChainLog || chain.count > chain.log_size) throw Error(ZS_EGENERIC, "fold chain size");
  k_fold_chain<<<1, kChainThreads, 0, st>>>(chain);
  ZS_CUDA(cudaGetLastError());
}

// One node per thread at the first layer's widest level; the levels are then chains of two
// compressions (1.3 us each), the transcript's step another two to four.
constexpr unsigned kTailThreads = kTailMax / 2;
__global__ void __launch_bounds__(kTailThreads) k_fri_tail(const FriTail* __restrict__ ftp, Channel* ch) {
  const FriTail& ft = *ftp;
  __shared__ wtx::Shared s_tx;
  __shared__ uint4 s_dig[2 * 3 * (kTailMax / 4)];
  __shared__ qm31 s_c;  // the next fold's alpha * off_inv
  after_previous();
  if (threadIdx.x < 32) wtx::load(s_tx, ch);
  if (threadIdx.x == 0 && ft.layer[0]) s_c = qmul(ft.alphas[-1], ft.off_inv[0]);
  __syncthreads();
#pragma unroll 1
  for (uint32_t c = 0; c < ft.count; ++c) {
    const unsigned lg = ft.log_size - c;
    const FoldSource f{ft.layer[c], ft.layer[c + 1], nullptr, ft.tables, qzero(), 1u << lg, ft.first + c - 1};
    const qm31 fold_c = s_c;
    cta_levels<kFold>(ft.tree[c], lg, 0, lg, lg, 0, s_dig, ft.layer[c + 1], f, fold_c);  // ends with a barrier
    if (threadIdx.x < 32) {
      const uint32_t* root = ft.tree[c] + 8 * (((size_t)2 << lg) - 2);
      const qm31 alpha = wtx::step(s_tx, root);
      if (threadIdx.x < 8) ft.roots[8 * c + threadIdx.x] = __ldcg(root + threadIdx.x);
      if (threadIdx.x == 0) {
        ft.alphas[c] = alpha;
        s_c = qmul(alpha, ft.off_inv[c + 1]);
      }
    }
    __syncthreads();
  }
  if (threadIdx.x < 32) wtx::store(s_tx, ch);
  const uint32_t half = 1u << (ft.log_size - ft.count);
  const uint4* in = reinterpret_cast<const uint4*>(ft.layer[ft.count]);
  for (uint32_t j = threadIdx.x; j < half; j += blockDim.x)
    reinterpret_cast<uint4*>(ft.layer[ft.count + 1])[j] = u4_of(
        fold_value(q_of(__ldcg(in + j)), q_of(__ldcg(in + j + half)), j, ft.first + ft.count - 1, s_c, ft.tables));
}

void fri_tail(const FriTail* ft, Channel* ch, cudaStream_t st) {
  void* args[] = {&ft, &ch};
  launch_overlapped((const void*)k_fri_tail, dim3(1), dim3(kTailThreads), args, 0, st);
}

}  // namespace zs
