// NTTs over QM31 for the low-degree extension, computed in the CRT domain.
//
// QM31 = CM31[j]/(j^2 + i), and -i = s^2 with s = 2^15 (1 - i), so
//   phi: a + b j  ->  (a + b s, a - b s)
// is a ring isomorphism QM31 -> CM31 x CM31. Both components of the 2-adic root have
// order 2^32, so a DFT over a 2-power subgroup of QM31 is two CM31 DFTs with the
// component roots: every butterfly costs two CM31 products (3 M31 products each)
// instead of one QM31 product (9). phi and its inverse
//   a = (u + v) / 2,  b = (u - v) / (2 s) = (u - v)(1 + i) 2^-17
// are additions and rotations of the 31-bit word. The transform is exact, so its
// results equal the reference's Lagrange interpolation / Horner evaluation value for
// value (the DFT over the subgroup is invertible in both components).
//
// The second component is held conjugated: phi'(a + b j) = (a + b s, conj(a - b s)).
// Conjugation is an automorphism of CM31, so it changes the roots and nothing else, and both
// components' 4th root is then i and their 8th roots are (1 + i) 2^15 and -(1 + i) 2^15
// (NttTables checks this): a radix-8 butterfly takes its inner roots by additions and a
// rotation, the same instructions for both components, the sign swapping two outputs.
//
// The LDE: the inverse transform on H runs decimation-in-frequency (natural-order
// values in, bit-reversed coefficients out), so the zero-padded input of the forward
// decimation-in-time transform is written contiguously and its output is in natural
// order; neither needs a separate bit-reversal pass. Each transform is a few passes over
// HBM of up to 9 bits of the index (k_ntt_pass), three stages in registers at a time;
// the results enter and leave the CRT domain in the passes' loads and stores.
#include <algorithm>
#include <vector>

#include "ntt.cuh"

namespace zs {

namespace {
constexpr unsigned kThreads = 256;

__device__ __forceinline__ qm31 ldq(const qm31* p) {
  const uint4 r = *reinterpret_cast<const uint4*>(p);
  return qmake(r.x, r.y, r.z, r.w);
}
__device__ __forceinline__ void stq(qm31* p, const qm31& v) {
  *reinterpret_cast<uint4*>(p) = make_uint4(v.a.a, v.a.b, v.b.a, v.b.b);
}
__device__ __forceinline__ cm31 cshl(cm31 x, unsigned k) { return {mshl(x.a, k), mshl(x.b, k)}; }
ZS_HD cm31 cconj(cm31 x) { return {x.a, mneg(x.b)}; }
// The CRT image phi' of a QM31 value, held in the a and b slots of a qm31.
ZS_HD qm31 to_crt(const qm31& x) {
  // b s = 2^15 (1 - i)(c + d i) = 2^15 ((c + d) + (d - c) i)
  const cm31 bs = {mshl(madd(x.b.a, x.b.b), 15), mshl(msub(x.b.b, x.b.a), 15)};
  return {cadd(x.a, bs), cconj(csub(x.a, bs))};
}
// x t for a twiddle held doubled, T = 2 t (both words below 2^32): the sums of two products
// are 2 v < 2^64, whose high word is at >> 31 and at most 2p, and whose low word is 2 (v & p).
// Three ALU operations a word against seven for three reduced products and their sums.
// Inside a pass a word may be p for 0: sums, differences and products of words <= p are
// again <= p, and mshl, which ends every way out of the domain, gives 0 for it.
__device__ __forceinline__ uint32_t fold2(uint64_t x) {
  const uint32_t hi = (uint32_t)(x >> 32), h = umin32(hi, hi - P);
  const uint32_t r = h + ((uint32_t)x >> 1);
  return umin32(r, r - P);
}
__device__ __forceinline__ cm31 mul_tw(cm31 x, cm31 T) {
  const uint32_t nb = P - x.b;
  return {fold2((uint64_t)x.a * T.a + (uint64_t)nb * T.b), fold2((uint64_t)x.a * T.b + (uint64_t)x.b * T.a)};
}
__device__ __forceinline__ qm31 twice(const qm31& v) { return qmake(v.a.a << 1, v.a.b << 1, v.b.a << 1, v.b.b << 1); }
// Products with the 4th root i and its inverse, and with the 8th root (1 + i) 2^15 and its
// inverse (1 - i) 2^15 (the first component's; the second's have the other sign).
__device__ __forceinline__ cm31 mul_w4(cm31 x) { return {P - x.b, x.a}; }
__device__ __forceinline__ cm31 mul_w4i(cm31 x) { return {x.b, P - x.a}; }
__device__ __forceinline__ uint32_t rot15(uint32_t x) { return ((x << 15) | (x >> 16)) & P; }  // x 2^15
__device__ __forceinline__ cm31 mul_w8(cm31 x) { return {rot15(msub(x.a, x.b)), rot15(madd(x.a, x.b))}; }
__device__ __forceinline__ cm31 mul_w8i(cm31 x) { return {rot15(madd(x.a, x.b)), rot15(msub(x.b, x.a))}; }
}  // namespace

// pows[k] = x^k: each thread raises x to its first index, then multiplies along a
// run of kPowRun consecutive powers.
constexpr uint32_t kPowRun = 16;
__global__ void k_qpowers(qm31 x, qm31* pows, uint32_t count) {
  const uint32_t k0 = (blockIdx.x * blockDim.x + threadIdx.x) * kPowRun;
  if (k0 >= count) return;
  qm31 v = qpow(x, k0);
  for (uint32_t k = k0; k < count && k < k0 + kPowRun; ++k) {
    stq(pows + k, v);
    v = qmul(v, x);
  }
}

void qm31_powers(qm31 x, qm31* pows, uint32_t count, cudaStream_t st) {
  if (count == 0) return;
  const uint32_t threads = (count + kPowRun - 1) / kPowRun;
  k_qpowers<<<(threads + kThreads - 1) / kThreads, kThreads, 0, st>>>(x, pows, count);
  ZS_CUDA(cudaGetLastError());
}

// out = 2 phi'(in), the tables' form
__global__ void k_to_crt(const qm31* in, qm31* out, uint32_t count) {
  const uint32_t k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) stq(out + k, twice(to_crt(ldq(in + k))));
}

NttTables::NttTables(unsigned l, cudaStream_t s) : log_n(l), st(s) {
  if (log_n > 30) throw Error(ZS_EMALFORMED, "NTT size above 2^30");
  {  // the passes' inner roots
    const qm31 w4 = to_crt(q_root_of_unity(2)), w8 = to_crt(q_root_of_unity(3));
    const uint32_t h = 1u << 15;
    if (!qeq(w4, qmake(0, 1, 0, 1)) || !qeq(w8, qmake(h, h, P - h, P - h)))
      throw Error(ZS_EGENERIC, "unexpected CRT images of the 4th and 8th roots of unity");
  }
  const uint32_t half = log_n == 0 ? 1 : (1u << (log_n - 1));
  ZS_CUDA(cudaMallocAsync(&fwd, half * sizeof(qm31), st));
  ZS_CUDA(cudaMallocAsync(&inv_crt, half * sizeof(qm31), st));
  ZS_CUDA(cudaMallocAsync(&fwd_crt, half * sizeof(qm31), st));
  const qm31 w = q_root_of_unity(log_n);
  qm31_powers(w, fwd, half, st);
  k_to_crt<<<(half + kThreads - 1) / kThreads, kThreads, 0, st>>>(fwd, fwd_crt, half);
  qm31_powers(qinv(w), inv_crt, half, st);
  k_to_crt<<<(half + kThreads - 1) / kThreads, kThreads, 0, st>>>(inv_crt, inv_crt, half);
  ZS_CUDA(cudaGetLastError());
}
NttTables::~NttTables() {
  cudaFreeAsync(fwd, st);
  cudaFreeAsync(fwd_crt, st);
  cudaFreeAsync(inv_crt, st);
}

// out[j] = 2 phi'(offset^bitrev(j)) for j < 2^log_n, `in` the powers in natural order.
__global__ void k_to_crt_brev(const qm31* __restrict__ in, qm31* __restrict__ out, unsigned log_n) {
  const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j < (1u << log_n)) stq(out + j, twice(to_crt(ldq(in + bitrev(j, log_n)))));
}

OffsetTable::OffsetTable(unsigned log_n, cudaStream_t s) : st(s) {
  const uint32_t n = 1u << log_n;
  qm31* pows = nullptr;
  ZS_CUDA(cudaMallocAsync(&pows, n * sizeof(qm31), st));
  ZS_CUDA(cudaMallocAsync(&crt, n * sizeof(qm31), st));
  qm31_powers(q_fri_offset(), pows, n, st);
  k_to_crt_brev<<<(n + kThreads - 1) / kThreads, kThreads, 0, st>>>(pows, crt, log_n);
  ZS_CUDA(cudaGetLastError());
  ZS_CUDA(cudaFreeAsync(pows, st));
}
OffsetTable::~OffsetTable() { cudaFreeAsync(crt, st); }

// One pass of a size-2^logN transform: the stages of index bits [lo, lo + M), for `count`
// columns (blockIdx.y). An index is j = hi << (lo + M) | mid << lo | l; a CTA takes all mid
// of 2^lgG consecutive l and 2^lgH consecutive hi (more than one only where l is whole, so
// that its elements are contiguous): 2^E elements, e = hi | mid | l, E = lgG + M + lgH.
//
// A thread works on one component of eight elements (16 registers), lanes 2i and 2i + 1 on
// the two components of the same ones, so that a warp reads and writes whole elements. The
// stages go in chunks of up to three, each on eight elements that differ in three bits of e
// starting at the chunk's lowest; between chunks the elements change threads through shared
// memory (8-byte slots, two of padding per 16: conflict-free for every position of the three
// bits). The first chunk reads global memory into registers and the last writes it from
// there. An earlier form kept the elements in shared memory, two stages per round trip with
// their twiddles staged there too, and waited on it (issue slots 42-53 % busy).
//
// Stages s of a chunk at bits [b, b + R) of mid, all in one (DIT; DIF is its transpose):
//   y_q = sum_m w_{2^R}^(q rev(m)) T^(k rev(m)) x_m,  T = w_{2^(lo+b+R)}, k = the index bits
// below the chunk: 2^R - 1 products by loaded twiddles, then a DFT whose roots are 1, i and
// (1 + i) 2^15, free of products.
//
// Where the first pass reads: kInPlace `a`; kToCrt QM31 values of `src`, mapped into the CRT
// domain; kExpand `src[j >> lo]`, the compact CRT values whose 2^lo copies the stages below
// of a zero-padded DIT would make. Where the last one writes: kCrt `a`; kQm31 `a`, out of
// the CRT domain; kCoeffs (inverse) the values times 1/N = 2^sh out of the CRT domain to `a`
// and times offset^bitrev(j) to `wbuf`, the forward transform's compact input.
enum InMode : unsigned { kInPlace = 0, kToCrt = 1, kExpand = 2 };
enum OutMode : unsigned { kCrt = 0, kQm31 = 1, kCoeffs = 2 };
struct NttPass {
  qm31* a;
  size_t stride;
  const qm31* src;
  size_t src_stride;
  const qm31* tw;
  const qm31* offset_crt;
  qm31* wbuf;
  size_t w_stride;
  unsigned in_mode, out_mode, logN, lo, M, lgG, lgH;
};

// Component c of a table's entry: the tables are written before any pass is launched.
__device__ __forceinline__ cm31 ldc(const qm31* p, uint32_t c) {
  const uint2 r = __ldg(reinterpret_cast<const uint2*>(p) + c);
  return {r.x, r.y};
}
// Component c of what an earlier pass wrote, which may end while this one's CTAs are up: a
// plain load, never the read-only path (launch_overlapped).
__device__ __forceinline__ cm31 ld_pass(const qm31* p, uint32_t c) {
  const uint2 r = reinterpret_cast<const uint2*>(p)[c];
  return {r.x, r.y};
}

// 2 w^i of component c for i < N, from the table of i < N/2 (w^(N/2) = -1); `wraps`: i may
// reach N/2.
__device__ __forceinline__ cm31 twiddle(const qm31* __restrict__ tw, uint32_t i, uint32_t half, bool wraps,
                                        uint32_t c) {
  if (!wraps) return ldc(tw + i, c);
  const bool neg = i >= half;
  const cm31 t = ldc(tw + (neg ? i - half : i), c);
  return neg ? cm31{2 * P - t.a, 2 * P - t.b} : t;
}

// The R stages of a chunk on the elements' bits [D, D + R) of the eight in v. k0: the index
// bits below the eight elements' lowest bit; bit_k: what each of the D element bits below the
// chunk adds to k. sh: logN - (lo + b + R).
template <bool DIF, int R, int D>
__device__ __forceinline__ void chunk8(cm31 (&v)[8], const qm31* __restrict__ tw, unsigned logN, unsigned sh,
                                       uint32_t k0, uint32_t bit_k, bool unit, uint32_t c) {
  const uint32_t half = 1u << (logN - 1);
  constexpr int Q = 1 << R;
  auto rev = [](int m) { return R == 3 ? ((m & 1) << 2) | (m & 2) | (m >> 2) : R == 2 ? ((m & 1) << 1) | (m >> 1) : m; };
  // element index of transform index m in group g (g: the three bits without [D, D + R))
  auto at = [](int g, int m) { return (g & ((1 << D) - 1)) | (m << D) | ((g >> D) << (D + R)); };
  auto twiddles = [&] {
    if (unit) return;  // k = 0 throughout
#pragma unroll
    for (int m = 1; m < Q; ++m) {
#pragma unroll
      for (int glo = 0; glo < (1 << D); ++glo) {  // the groups that share k
        // k << sh < N / 2^R, so only multiples above 2^(R-1) wrap
        const uint32_t k = (k0 + glo * bit_k) << sh;
        const cm31 t = twiddle(tw, k * rev(m), half, 2 * rev(m) > Q, c);
#pragma unroll
        for (int ghi = 0; ghi < (8 >> (R + D)); ++ghi) {
          cm31& x = v[at(glo | (ghi << D), m)];
          x = mul_tw(x, t);
        }
      }
    }
  };
  if (!DIF) twiddles();
#pragma unroll
  for (int g = 0; g < 8 / Q; ++g) {
#pragma unroll
    for (int s = 0; s < R; ++s) {
      const int bit = DIF ? R - 1 - s : s;
#pragma unroll
      for (int m = 0; m < Q; ++m) {
        if (m & (1 << bit)) continue;
        cm31 &x = v[at(g, m)], &y = v[at(g, m | (1 << bit))];
        const int q = m & ((1 << bit) - 1);  // the root w_{2^(bit+1)}^q: 1; i; (1 + i) 2^15 and its powers
        if (!DIF) {
          cm31 t = y;
          if (bit == 1 && q == 1) t = mul_w4(y);
          if (bit == 2 && q == 1) t = mul_w8(y);
          if (bit == 2 && q == 2) t = mul_w4(y);
          if (bit == 2 && q == 3) t = mul_w8(mul_w4(y));
          y = csub(x, t);
          x = cadd(x, t);
        } else {
          const cm31 d = csub(x, y);
          x = cadd(x, y);
          y = d;
          if (bit == 1 && q == 1) y = mul_w4i(d);
          if (bit == 2 && q == 1) y = mul_w8i(d);
          if (bit == 2 && q == 2) y = mul_w4i(d);
          if (bit == 2 && q == 3) y = mul_w8i(mul_w4i(d));
        }
      }
    }
  }
  if (DIF) twiddles();
}

// Bound by integer issue (40-50 instructions an element and stage, 26 by count; ALU pipe 60-74 %)
// and by the latency of the twiddle loads. Three stages between two trips through shared memory,
// products summed in 64 bits, the ways in and out of the CRT domain in the loads and stores:
// the transforms of a 387-column linear layer of 2^15 rows 3221 -> 2560 us, of a stacked Rescue
// proof of 2^18 rows 914 -> 698 us, against two stages a trip and separate passes.
constexpr unsigned kTileLog = 11;  // elements of a CTA's tile: 32 KB, 512 threads
__device__ __forceinline__ uint32_t slot_of(uint32_t e, uint32_t c) {
  const uint32_t s = 2 * e + c;
  return s + 2 * (s >> 4);
}

template <bool DIF>
__global__ void __launch_bounds__(1 << (kTileLog - 2), 2) k_ntt_pass(const __grid_constant__ NttPass p) {
  extern __shared__ uint2 s_el[];
  let_next_start();
  after_previous();
  const unsigned E = p.lgG + p.M + p.lgH, lo = p.lo, M = p.M;
  const uint32_t c = threadIdx.x & 1, q = threadIdx.x >> 1;
  // the tile: l0 = the first l, hi0 = the first hi
  const uint32_t l_tiles = 1u << (lo - p.lgG);
  const uint32_t l0 = (blockIdx.x & (l_tiles - 1)) << p.lgG, hi0 = (blockIdx.x >> (lo - p.lgG)) << p.lgH;
  qm31* col = p.a + (size_t)blockIdx.y * p.stride;
  // the element's index in the transform; both it and the shared-memory slot are sums over
  // the bits of e
  const uint32_t tile = (hi0 << (lo + M)) | l0;
  auto index = [&](uint32_t e) { return tile + ((e >> p.lgG) << lo) + (e & ((1u << p.lgG) - 1)); };
  // the lowest chunk takes what is left; M = 0 (only copies) has one without stages
  const unsigned n_chunks = max(1u, (M + 2) / 3), first = M - 3 * (n_chunks - 1);
  cm31 v[8];
#pragma unroll 1
  for (unsigned i = 0; i < n_chunks; ++i) {
    const unsigned ci = DIF ? n_chunks - 1 - i : i;
    const unsigned R = ci == 0 ? first : 3, b = ci == 0 ? 0 : first + 3 * (ci - 1);
    const unsigned pos = p.lgG + b, ws = min(pos, E - 3), D = pos - ws;
    // element m of this thread: e0 + (m << ws); with R = 3 the second component's odd ones
    // lie four further (mod 8): its 8th root has the other sign
    const uint32_t e0 = ((q >> ws) << (ws + 3)) | (q & ((1u << ws) - 1));
    const bool last = i + 1 == n_chunks;
    const bool pairs = last && ws > 0 && p.out_mode != kCrt;  // stored as whole elements by lane pairs
    const uint32_t swap = R == 3 && !(pairs && !DIF) ? c << 2 : 0;
    // at(base, w, m, swapped): base plus the weights w of the bits of element m
    struct W {
      uint32_t w[3], sw;
    };
    auto weights = [&](auto&& f) {
      W r{{f(1u << ws), f(2u << ws), f(4u << ws)}, 0};
      r.sw = swap ? r.w[2] : 0;
      return r;
    };
    auto at = [](uint32_t base, const W& w, int m, bool swapped) {
      const uint32_t o = base + (m & 1 ? w.w[0] : 0) + (m & 2 ? w.w[1] : 0) + (m & 4 ? w.w[2] : 0);
      return swapped && (m & 1) ? (m & 4 ? o - w.sw : o + w.sw) : o;
    };
    const W gw = weights([&](uint32_t e) { return index(e) - tile; });
    const W sw = weights([&](uint32_t e) { return slot_of(e, 0); });
    const uint32_t g0 = index(e0), s0 = slot_of(e0, c);
    if (i == 0) {
      const qm31* src = p.src + (size_t)blockIdx.y * p.src_stride;
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const uint32_t j = at(g0, gw, m, DIF);
        if (p.in_mode == kToCrt) {
          const qm31 x = to_crt(ldq(src + j));
          v[m] = c ? x.b : x.a;
        } else if (p.in_mode == kExpand) {
          v[m] = ld_pass(src + (j >> lo), c);
        } else {
          v[m] = ld_pass(col + j, c);
        }
      }
    } else {
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const uint2 r = s_el[at(s0, sw, m, DIF)];
        v[m] = {r.x, r.y};
      }
    }
    const uint32_t low = e0 & ((1u << pos) - 1);  // the bits of e below the eight elements' (D = 0)
    const uint32_t k0 = ((low >> p.lgG) << lo) | (l0 + (low & ((1u << p.lgG) - 1)));
    // for D > 0 (then b = 0) the bits [ws, pos) of l are element bits
    const uint32_t bit_k = 1u << ws;
    const unsigned sh = p.logN - (lo + b + R);
    const bool unit = lo + b == 0;
    if (R == 3) {
      chunk8<DIF, 3, 0>(v, p.tw, p.logN, sh, k0, 0, unit, c);
    } else if (R == 2) {
      if (D == 0) chunk8<DIF, 2, 0>(v, p.tw, p.logN, sh, k0, 0, unit, c);
      else chunk8<DIF, 2, 1>(v, p.tw, p.logN, sh, k0, bit_k, unit, c);
    } else if (R == 1) {
      if (D == 0) chunk8<DIF, 1, 0>(v, p.tw, p.logN, sh, k0, 0, unit, c);
      else if (D == 1) chunk8<DIF, 1, 1>(v, p.tw, p.logN, sh, k0, bit_k, unit, c);
      else chunk8<DIF, 1, 2>(v, p.tw, p.logN, sh, k0, bit_k, unit, c);
    }
    if (!DIF && pairs && R == 3) {  // the odd elements' exchange in registers instead
#pragma unroll
      for (int m = 1; m < 4; m += 2) {
        const cm31 x = v[m], y = v[m + 4];
        v[m] = c ? y : x, v[m + 4] = c ? x : y;
      }
    }
    if (!last || ws == 0) {  // (eight consecutive elements per thread: stored by rows below)
#pragma unroll
      for (int m = 0; m < 8; ++m) s_el[at(s0, sw, m, !DIF)] = make_uint2(v[m].a, v[m].b);
      __syncthreads();
    }
    if (!last) continue;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      uint32_t j = at(g0, gw, m, !DIF);
      cm31 x = v[m];
      if (ws == 0) {
        const uint32_t e = ((uint32_t)m << (E - 3)) | q;
        const uint2 r = s_el[slot_of(e, c)];
        x = {r.x, r.y};
        j = index(e);
      }
      if (p.out_mode == kCoeffs) {
        const unsigned rot = (31 - p.logN) % 31;  // 1/N = 2^(31 - logN)
        x = {mshl(x.a, rot), mshl(x.b, rot)};
        const cm31 w = mul_tw(x, ldc(p.offset_crt + j, c));
        reinterpret_cast<uint2*>(p.wbuf + (size_t)blockIdx.y * p.w_stride + j)[c] = make_uint2(w.a, w.b);
      }
      if (p.out_mode != kCrt) {
        // a = (u + v) / 2, b = (u - v) (1 + i) 2^-17, u and v in the lane pair (v conjugated)
        const cm31 mine = c ? cconj(x) : x;
        const cm31 other = {__shfl_xor_sync(0xffffffffu, mine.a, 1), __shfl_xor_sync(0xffffffffu, mine.b, 1)};
        if (c == 0) {
          x = cshl(cadd(mine, other), 30);  // 2^30 = 1/2
        } else {
          const cm31 d = csub(other, mine);
          x = {mshl(msub(d.a, d.b), 14), mshl(madd(d.a, d.b), 14)};
        }
      }
      reinterpret_cast<uint2*>(col + j)[c] = make_uint2(x.a, x.b);
    }
  }
}

// Transforms of fewer than eight elements (and of none), one thread per column: the sums
// themselves. DIF: x_q -> sum_m tw^(q m) x_m at bitrev(q); DIT: bit-reversed input.
template <bool DIF>
__global__ void k_ntt_tiny(const __grid_constant__ NttPass p, uint32_t count) {
  const uint32_t col_i = blockIdx.x * blockDim.x + threadIdx.x;
  if (col_i >= count) return;
  const uint32_t n = 1u << p.logN, half = n >> 1;
  qm31 x[4], y[4];
  for (uint32_t j = 0; j < n; ++j) {
    const qm31* src = p.in_mode == kInPlace ? p.a + (size_t)col_i * p.stride : p.src + (size_t)col_i * p.src_stride;
    const qm31 r = ldq(src + (p.in_mode == kExpand ? j >> p.lo : j));
    x[j] = p.in_mode == kToCrt ? to_crt(r) : r;
  }
  for (uint32_t o = 0; o < n; ++o) {
    y[o] = qzero();
    for (uint32_t j = 0; j < n; ++j) {
      // DIT copies below bit `lo`: the padded zeros are left out
      if (!DIF && (j & ((1u << p.lo) - 1))) continue;
      const uint32_t e = DIF ? (bitrev(o, p.logN) * j) & (n - 1) : (o * bitrev(j, p.logN)) & (n - 1);
      qm31 t = n == 1 ? twice(to_crt(qone())) : ldq(p.tw + (e >= half ? e - half : e));
      if (n > 1 && e >= half) t = qmake(2 * P - t.a.a, 2 * P - t.a.b, 2 * P - t.b.a, 2 * P - t.b.b);
      y[o] = {cadd(y[o].a, mul_tw(x[j].a, t.a)), cadd(y[o].b, mul_tw(x[j].b, t.b))};
    }
  }
  for (uint32_t j = 0; j < n; ++j) {
    qm31 v = y[j];
    if (p.out_mode == kCoeffs) {
      const unsigned rot = (31 - p.logN) % 31;
      v = {cshl(v.a, rot), cshl(v.b, rot)};
      const qm31 o = ldq(p.offset_crt + j);
      stq(p.wbuf + (size_t)col_i * p.w_stride + j, qm31{mul_tw(v.a, o.a), mul_tw(v.b, o.b)});
    }
    if (p.out_mode != kCrt) {
      const cm31 u = v.a, w = cconj(v.b), d = csub(u, w);
      v = {cshl(cadd(u, w), 30), {mshl(msub(d.a, d.b), 14), mshl(madd(d.a, d.b), 14)}};
    }
    stq(p.a + (size_t)col_i * p.stride + j, v);
  }
}

// The passes of a transform's bits [from, logN), lowest first: as few as 9 bits a pass
// allow, of even size. A pass takes 2^2 to 2^5 consecutive l where there are as many (64
// bytes and more per row), and whole blocks of contiguous elements otherwise.
static std::vector<NttPass> plan_passes(const NttPass& base, unsigned from) {
  std::vector<NttPass> v;
  const unsigned bits = base.logN - from, count = std::max(1u, (bits + 8) / 9);
  unsigned lo = from;
  for (unsigned i = 0; i < count; ++i) {
    NttPass p = base;
    p.lo = lo;
    p.M = (base.logN - lo + (count - i) - 1) / (count - i);
    p.lgG = std::min(lo, kTileLog - p.M);
    p.lgH = p.lgG == lo ? std::min(base.logN - lo - p.M, kTileLog - p.M - p.lgG) : 0;
    v.push_back(p);
    lo += p.M;
  }
  return v;
}

// The transform of `count` columns: bits [from, logN) (forward: those below only copy).
template <bool DIF>
static void run_transform(const NttPass& t, unsigned from, uint32_t count, cudaStream_t st) {
  if (t.logN < 3) {
    NttPass p = t;
    p.lo = from;
    k_ntt_tiny<DIF><<<(count + 63) / 64, 64, 0, st>>>(p, count);
    ZS_CUDA(cudaGetLastError());
    return;
  }
  std::vector<NttPass> plan = plan_passes(t, from);
  const size_t n = plan.size();
  for (size_t i = 0; i < n; ++i) {
    NttPass p = plan[DIF ? n - 1 - i : i];
    if (i > 0) p.in_mode = kInPlace, p.src = p.a, p.src_stride = p.stride;
    if (i + 1 < n) p.out_mode = kCrt;
    const unsigned E = p.lgG + p.M + p.lgH;
    const size_t smem = ((size_t)18 << E) / 8 * sizeof(uint2) + 16 * sizeof(uint2);
    for (uint32_t c0 = 0; c0 < count; c0 += 65535) {  // grid.y is at most 65535
      NttPass g = p;
      g.a += c0 * g.stride, g.src += c0 * g.src_stride, g.wbuf += g.wbuf ? c0 * g.w_stride : 0;
      void* args[] = {&g};
      launch_overlapped((const void*)k_ntt_pass<DIF>, dim3(1u << (p.logN - E), std::min(65535u, count - c0)),
                        dim3(1u << (E - 2)), args, smem, st);
    }
  }
  ZS_CUDA(cudaGetLastError());
}

void lde_qm31(const qm31* values, size_t v_stride, qm31* coeffs, size_t c_stride, qm31* codeword, size_t w_stride,
              uint32_t C, const NttTables& small, const NttTables& big, const OffsetTable& offset, cudaStream_t st) {
  const unsigned log_n = small.log_n, log_N = big.log_n;
  const uint32_t n = 1u << log_n;
  if (log_N == 0) throw Error(ZS_EMALFORMED, "LDE onto a domain of one point");
  qm31* wbuf = nullptr;
  ZS_CUDA(cudaMallocAsync((void**)&wbuf, (size_t)C * n * sizeof(qm31), st));
  // inverse transform on H: natural-order values in, bit-reversed coefficients out, and the
  // coefficients times offset^k, the forward transform's input, in `wbuf`
  NttPass inv{};
  inv.a = coeffs, inv.stride = c_stride, inv.src = values, inv.src_stride = v_stride, inv.tw = small.inv_crt;
  inv.offset_crt = offset.crt, inv.wbuf = wbuf, inv.w_stride = n;
  inv.in_mode = kToCrt, inv.out_mode = kCoeffs, inv.logN = log_n;
  run_transform<true>(inv, 0, C, st);
  // phi'(c_k offset^k) belongs at position bitrev_N(k) = j << B of the size-N input, j its
  // place in `wbuf`; the input is zero elsewhere, so the first B stages only copy
  NttPass fwd{};
  fwd.a = codeword, fwd.stride = w_stride, fwd.src = wbuf, fwd.src_stride = n, fwd.tw = big.fwd_crt;
  fwd.in_mode = kExpand, fwd.out_mode = kQm31, fwd.logN = log_N;
  run_transform<false>(fwd, log_N - log_n, C, st);
  ZS_CUDA(cudaFreeAsync(wbuf, st));
}

}  // namespace zs
