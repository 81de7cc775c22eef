// The levels of Merkle trees inside one CTA (device code of merkle.cu and fri.cu).
#pragma once
#include "blake3.cuh"
#include "common.cuh"
#include "merkle.cuh"

namespace zs {

__device__ __forceinline__ void put_digest(uint32_t* tree_words, size_t digest_index, const uint32_t o[8]) {
  uint4* dst = reinterpret_cast<uint4*>(tree_words + 8 * digest_index);
  dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
  dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

__device__ __forceinline__ qm31 q_of(const uint4& r) { return qmake(r.x, r.y, r.z, r.w); }
__device__ __forceinline__ uint4 u4_of(const qm31& v) { return make_uint4(v.a.a, v.a.b, v.b.a, v.b.b); }

// Where a subtree's lowest level comes from: digests of level `level0` in the tree; the
// values of a layer, hashed to leaves; or a fold of the layer before (kFold with a null
// `in` takes values), whose outputs are stored as well.
enum TreeSource : int { kDigests = 0, kValues = 1, kFold = 2 };

// x/2 mod p
__device__ __forceinline__ uint32_t mhalf(uint32_t x) { return (x >> 1) | ((x & 1) << 30); }

// One value of a fold (fri.zig:209-219): with x = D_layer[j],
//   (y0 + y1) / 2 + alpha (y0 - y1) / (2 x) = ((y0 + y1) + (y0 - y1) c w_0^-(j 2^layer)) / 2,
// c = alpha FRI_OFFSET^-(2^layer), the power of w_0^-1 from the fold tables.
__device__ __forceinline__ qm31 fold_value(const qm31& y0, const qm31& y1, uint32_t j, unsigned layer, const qm31& c,
                                           const qm31* __restrict__ tables) {
  const uint4* t = reinterpret_cast<const uint4*>(tables);
  const uint64_t k = (uint64_t)j << layer;
  qm31 w = qmul(q_of(__ldg(t + (k & 2047))), q_of(__ldg(t + 2048 + ((k >> 11) & 2047))));
  if (k >> 22) w = qmul(w, q_of(__ldg(t + 4096 + ((k >> 22) & 2047))));
  const qm31 r = qadd(qadd(y0, y1), qmul(qsub(y0, y1), qmul(w, c)));
  return qmake(mhalf(r.a.a), mhalf(r.a.b), mhalf(r.b.a), mhalf(r.b.b));
}

// Levels level0 + 1 .. level0 + levels of a tree of 2^log_n leaves over the 2^span digests
// [cta 2^span, (cta + 1) 2^span) of level `level0`, one node per thread, a barrier between
// levels (of the warp where one suffices) and one at the end; kValues and kFold (level0 = 0) hash those digests first, two
// leaves to a node. All levels run through one loop with one copy of hash2: a copy is 26 KB
// of instructions, and the seven copies of an earlier kernel (a 3-level subtree per thread)
// ran at the rate of the instruction cache, not of the ALU.
// s_dig: the digests of the last level, two levels in turn (3 * 2^(span - 2) digests).
template <int SRC>
__device__ __forceinline__ void cta_levels(uint32_t* words, unsigned log_n, unsigned level0, unsigned span,
                                           unsigned levels, size_t cta, uint4* s_dig, const qm31* vals,
                                           const FoldSource& f, const qm31& fold_c) {
  const size_t N2 = (size_t)2 << log_n;
  uint32_t from = 0, to = 0;  // offsets of the two levels in s_dig, in digests
#pragma unroll 1
  for (unsigned l = 1; l <= levels; ++l) {
    const uint32_t cnt = 1u << (span - l);
    if (cnt < 32 && threadIdx.x >= 32) break;  // the last levels are the first warp's alone
    const size_t dst = (N2 - (N2 >> (level0 + l))) + (cta << (span - l));
    const bool leaves = SRC != kDigests && level0 == 0 && l == 1;
    // The children's digests (or their leaves' values) in `q`, loaded one node ahead: warps
    // that all hash alike reach their loads together, and nothing else covers them.
    const uint4* src = leaves   ? reinterpret_cast<const uint4*>(SRC == kFold && f.in ? f.in : vals) + (cta << span)
                       : l == 1 ? reinterpret_cast<const uint4*>(words + 8 * ((N2 - (N2 >> level0)) + (cta << span)))
                                : s_dig + 2 * from;
    uint4 q[4];
    auto load = [&](uint32_t e) {
      if (leaves) {
        q[0] = __ldcg(src + 2 * e), q[1] = __ldcg(src + 2 * e + 1);
        if (SRC == kFold && f.in) q[2] = __ldcg(src + f.half + 2 * e), q[3] = __ldcg(src + f.half + 2 * e + 1);
      } else if (l == 1) {  // past L1: other CTAs may have written them in this launch
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = __ldcg(src + 4 * e + k);
      } else {
#pragma unroll
        for (int k = 0; k < 4; ++k) q[k] = src[4 * e + k];
      }
    };
    if (threadIdx.x < cnt) load(threadIdx.x);
#pragma unroll 1
    for (uint32_t e = threadIdx.x; e < cnt; e += blockDim.x) {
      uint32_t lc[8] = {q[0].x, q[0].y, q[0].z, q[0].w, q[1].x, q[1].y, q[1].z, q[1].w};
      uint32_t rc[8] = {q[2].x, q[2].y, q[2].z, q[2].w, q[3].x, q[3].y, q[3].z, q[3].w};
      if (e + blockDim.x < cnt) load(e + blockDim.x);
      uint32_t o[8];
      if (leaves) {  // hash the two leaves first, the second into rc
        const size_t leaf = (cta << span) + 2 * (size_t)e;
        uint32_t v[4] = {lc[0], lc[1], lc[2], lc[3]}, h[8];
#pragma unroll 1
        for (int k = 0; k < 2; ++k) {
          qm31 x = qmake(v[0], v[1], v[2], v[3]);
          if (SRC == kFold && f.in) {
            x = fold_value(x, qmake(rc[0], rc[1], rc[2], rc[3]), (uint32_t)leaf + k, f.layer, fold_c, f.tables);
            reinterpret_cast<uint4*>(f.out)[leaf + k] = u4_of(x);
          }
          b3::hash_qm31(x, h);
          put_digest(words, leaf + k, h);
          if (k == 0) {
#pragma unroll
            for (int w = 0; w < 4; ++w) v[w] = lc[4 + w], rc[w] = rc[4 + w];
#pragma unroll
            for (int w = 0; w < 8; ++w) lc[w] = h[w];
          }
        }
#pragma unroll
        for (int w = 0; w < 8; ++w) rc[w] = h[w];
      }
      b3::hash2(lc, rc, o);
      put_digest(words, dst + e, o);
      if (l < levels) put_digest(reinterpret_cast<uint32_t*>(s_dig), to + e, o);
    }
    if (cnt < 32)
      __syncwarp();
    else
      __syncthreads();
    from = to;
    to = to == 0 ? 1u << (span - 1) : 0;
  }
  __syncthreads();
}

}  // namespace zs
