// The Fiat-Shamir transcript's step on the device: one warp absorbs a layer's root and
// samples the folding challenge (fri.zig:199-206), on a copy of the host's Channel in
// shared memory.
//
// A step is two to four compressions, each waiting for the one before. In one thread, with
// byte-wise state updates, it took 11.5 us; here the lanes move the bytes and every lane
// computes the compression, so nothing has to be exchanged between its rounds.
#pragma once
#include "host.cuh"

namespace zs {
#ifdef __CUDACC__
namespace wtx {

// out[0..8) = the chaining value of compress(cv, m, counter, len, flags), all in shared
// memory, by a converged warp. The rounds run in a loop (the message permuted between them,
// m'[i] = m[PERM[i]]): a step's code is cold, and 2 KB of it load faster than 13.
static __device__ __noinline__ void compress(const uint32_t* cv, const uint32_t* ms, uint64_t counter, uint32_t len,
                                             uint32_t flags, uint32_t* out) {
#ifdef __CUDA_ARCH__
  using namespace b3;
  uint32_t a[4], b[4], c[4] = {IV0, IV1, IV2, IV3}, d[4] = {(uint32_t)counter, (uint32_t)(counter >> 32), len, flags};
  uint32_t m[16];
#pragma unroll
  for (int i = 0; i < 4; ++i) a[i] = cv[i], b[i] = cv[4 + i];
#pragma unroll
  for (int i = 0; i < 16; ++i) m[i] = ms[i];
#pragma unroll 1
  for (int r = 0; r < 7; ++r) {
#pragma unroll
    for (int i = 0; i < 4; ++i) g_dev<false, false>(a[i], b[i], c[i], d[i], m[2 * i], m[2 * i + 1]);
#pragma unroll
    for (int i = 0; i < 4; ++i)
      g_dev<false, false>(a[i], b[(i + 1) & 3], c[(i + 2) & 3], d[(i + 3) & 3], m[8 + 2 * i], m[9 + 2 * i]);
    constexpr int perm[16] = {2, 6, 3, 10, 7, 0, 4, 13, 1, 11, 12, 5, 9, 14, 15, 8};
    uint32_t t[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) t[i] = m[perm[i]];
#pragma unroll
    for (int i = 0; i < 16; ++i) m[i] = t[i];
  }
  __syncwarp();  // `out` may be `cv` or part of `ms`
  if ((threadIdx.x & 31) == 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) out[i] = a[i] ^ c[i], out[4 + i] = b[i] ^ d[i];
  }
  __syncwarp();
#endif
}

// Shared memory of a step: the transcript, a snapshot of it, a parent node's message and
// the bytes being absorbed.
struct Shared {
  alignas(16) unsigned char ch[sizeof(Channel)];
  alignas(16) unsigned char snap[sizeof(Hasher)];
  uint32_t msg[16];
  uint32_t dig[8];
  uint32_t iv[8];
};
static_assert(sizeof(Hasher) % 4 == 0 && offsetof(Hasher, block) % 4 == 0, "the state is moved in words");

__device__ __forceinline__ uint32_t* block_words(Hasher& h) { return reinterpret_cast<uint32_t*>(h.block); }

// h.update(src, n) for bytes in shared memory (the statements of Hasher::update).
__device__ __forceinline__ void update(Shared& s, Hasher& h, const uint8_t* src, uint32_t n) {
  const uint32_t lane = threadIdx.x & 31;
  uint32_t done = 0;
  while (done < n) {
    uint32_t len = h.block_len;
    const uint32_t blocks = h.blocks_done;
    const uint32_t start = blocks == 0 ? b3::CHUNK_START : 0u;
    if (len == 64) {
      const bool chunk = blocks * 64 + len == 1024;
      compress(h.cv, block_words(h), h.chunk_counter, 64, start | (chunk ? b3::CHUNK_END : 0u), h.cv);
      if (chunk) {  // its chaining value goes on the stack, merged with the subtrees it completes
        uint64_t total = h.chunk_counter + 1;
        uint32_t depth = h.depth;
        __syncwarp();
        if (lane == 0) h.chunk_counter = total;
        for (; (total & 1) == 0; total >>= 1) {
          --depth;
          if (lane < 8) s.msg[lane] = h.stack[depth][lane], s.msg[8 + lane] = h.cv[lane];
          __syncwarp();
          compress(s.iv, s.msg, 0, 64, b3::PARENT, h.cv);
        }
        if (lane < 8) h.stack[depth][lane] = h.cv[lane];
        __syncwarp();
        if (lane < 8) h.cv[lane] = s.iv[lane];
        if (lane == 0) h.depth = depth + 1;
      }
      if (lane < 16) block_words(h)[lane] = 0;
      if (lane == 0) h.block_len = 0, h.blocks_done = chunk ? 0 : blocks + 1;
      __syncwarp();
      len = 0;
    }
    const uint32_t take = min(64 - len, n - done);
    for (uint32_t i = lane; i < take; i += 32) h.block[len + i] = src[done + i];
    __syncwarp();  // every lane has read block_len
    if (lane == 0) h.block_len = len + take;
    __syncwarp();
    done += take;
  }
}

// s.dig = h.finalize().
__device__ __forceinline__ void finalize(Shared& s, Hasher& h) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t flags = (h.blocks_done == 0 ? b3::CHUNK_START : 0u) | b3::CHUNK_END;
  const uint32_t depth = h.depth;
  compress(h.cv, block_words(h), h.chunk_counter, h.block_len, flags | (depth == 0 ? b3::ROOT : 0u), s.dig);
  for (uint32_t k = depth; k-- > 0;) {
    if (lane < 8) s.msg[lane] = h.stack[k][lane], s.msg[8 + lane] = s.dig[lane];
    __syncwarp();
    compress(s.iv, s.msg, 0, 64, b3::PARENT | (k == 0 ? b3::ROOT : 0u), s.dig);
  }
}

// Loads the transcript (the calling warp, converged).
__device__ __forceinline__ void load(Shared& s, const Channel* ch) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(ch);
  uint32_t* dst = reinterpret_cast<uint32_t*>(s.ch);
  for (uint32_t i = lane; i < sizeof(Channel) / 4; i += 32) dst[i] = __ldcg(src + i);
  constexpr uint32_t iv[8] = {b3::IV0, b3::IV1, b3::IV2, b3::IV3, b3::IV4, b3::IV5, b3::IV6, b3::IV7};
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < 8; ++i) s.iv[i] = iv[i];
  __syncwarp();
}
__device__ __forceinline__ void store(Shared& s, Channel* ch) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t* src = reinterpret_cast<const uint32_t*>(s.ch);
  uint32_t* dst = reinterpret_cast<uint32_t*>(ch);
  for (uint32_t i = lane; i < sizeof(Channel) / 4; i += 32) dst[i] = src[i];
  __syncwarp();
}

// Absorbs the 32 bytes at `root` and returns a sampled QM31 (in every lane).
__device__ __forceinline__ qm31 step(Shared& s, const uint32_t* root) {
  const uint32_t lane = threadIdx.x & 31;
  Hasher& h = reinterpret_cast<Channel*>(s.ch)->h;
  Hasher& snap = *reinterpret_cast<Hasher*>(s.snap);
  if (lane < 8) s.dig[lane] = __ldcg(root + lane);
  __syncwarp();
  update(s, h, reinterpret_cast<const uint8_t*>(s.dig), 32);
  // the sample: a snapshot absorbs "zig-stark:sample" and the counter 0
  const uint32_t live = offsetof(Hasher, stack) / 4 + 8 * h.depth;  // words up to the live stack's end
  for (uint32_t i = lane; i < live; i += 32)
    reinterpret_cast<uint32_t*>(&snap)[i] = reinterpret_cast<const uint32_t*>(&h)[i];
  if (lane == 0) snap.depth = h.depth;
  constexpr uint32_t label[6] = {0x2d67697au, 0x72617473u, 0x61733a6bu, 0x656c706du, 0u, 0u};
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < 6; ++i) s.dig[i] = label[i];
  __syncwarp();
  update(s, snap, reinterpret_cast<const uint8_t*>(s.dig), 24);
  finalize(s, snap);
  const qm31 r = qmake(s.dig[0], s.dig[1], s.dig[2], s.dig[3]);
  update(s, h, reinterpret_cast<const uint8_t*>(s.dig), 32);
  auto red = [](uint32_t v) {  // M31.fromBytes: v mod p, v < 2^32 <= 2p + 2
    v = v >= P ? v - P : v;
    return v >= P ? v - P : v;
  };
  return qmake(red(r.a.a), red(r.a.b), red(r.b.a), red(r.b.b));
}

}  // namespace wtx
#endif
}  // namespace zs
