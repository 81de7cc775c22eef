// Exact M31 / CM31 / QM31 arithmetic for host and device.
//
// Field tower of the reference: M31 = F_(2^31-1) (src/m31/field/m31.zig),
// CM31 = M31[i]/(i^2+1) (cm31.zig), QM31 = CM31[j]/(j^2+i) (qm31.zig).
// Every function returns the canonical representative in [0, p), the same value
// the reference computes, so results are bit-identical to it whatever the
// evaluation order (the tower is a commutative ring and all operations are exact).
//
// Reductions use one conditional subtraction expressed as an unsigned min:
//   add: a + b < 2p        -> min(s, s - p)
//   sub: a - b (mod 2^32)  -> min(d, d + p)
//   mul: (a*b & p) + (a*b >> 31) <= 2p - 3 for a, b < p -> min(s, s - p)
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define ZS_HD __host__ __device__ __forceinline__
#else
#define ZS_HD inline
#endif

namespace zs {

constexpr uint32_t P = 2147483647u;

ZS_HD uint32_t umin32(uint32_t a, uint32_t b) { return a < b ? a : b; }

ZS_HD uint32_t madd(uint32_t a, uint32_t b) {
  uint32_t s = a + b;
  return umin32(s, s - P);
}
ZS_HD uint32_t msub(uint32_t a, uint32_t b) {
  uint32_t d = a - b;
  return umin32(d, d + P);
}
ZS_HD uint32_t mneg(uint32_t a) { return a == 0 ? 0 : P - a; }
ZS_HD uint32_t mmul(uint32_t a, uint32_t b) {
  uint64_t prod = (uint64_t)a * (uint64_t)b;
  uint32_t s = ((uint32_t)prod & P) + (uint32_t)(prod >> 31);
  return umin32(s, s - P);
}
// x * 2^k mod p for 0 <= k < 31: a rotation inside the 31-bit word.
ZS_HD uint32_t mshl(uint32_t x, unsigned k) {
  uint32_t r = ((x << k) | (x >> (31 - k))) & P;
  return r == P ? 0 : r;
}
// a^(p-2); 0 maps to 0 exactly as the reference's release build does. By the addition chain
// 1, 2, 3, 6, 7, 14, 28, 29 on the exponents 2^k - 1, and p - 2 = 4 (2^29 - 1) + 1: 38
// products in place of binary exponentiation's 60 (stacked Rescue 2^18: quotient 197 -> 190 us,
// DEEP 110 -> 107 us, proof 3.88 -> 3.84 ms).
ZS_HD uint32_t minv(uint32_t a) {
  auto up = [](uint32_t x, int k) {  // x^(2^k)
    for (int i = 0; i < k; ++i) x = mmul(x, x);
    return x;
  };
  const uint32_t x2 = mmul(up(a, 1), a), x3 = mmul(up(x2, 1), a), x6 = mmul(up(x3, 3), x3);
  const uint32_t x7 = mmul(up(x6, 1), a), x14 = mmul(up(x7, 7), x7), x28 = mmul(up(x14, 14), x14);
  return mmul(up(mmul(up(x28, 1), a), 2), a);
}

struct cm31 {
  uint32_t a, b;  // a + b i
};
ZS_HD cm31 cadd(cm31 x, cm31 y) { return {madd(x.a, y.a), madd(x.b, y.b)}; }
ZS_HD cm31 csub(cm31 x, cm31 y) { return {msub(x.a, y.a), msub(x.b, y.b)}; }
ZS_HD cm31 cneg(cm31 x) { return {mneg(x.a), mneg(x.b)}; }
// Karatsuba: (a+bi)(c+di) = (ac - bd) + ((a+b)(c+d) - ac - bd) i.
ZS_HD cm31 cmul(cm31 x, cm31 y) {
  uint32_t ac = mmul(x.a, y.a), bd = mmul(x.b, y.b);
  uint32_t t = mmul(madd(x.a, x.b), madd(y.a, y.b));
  return {msub(ac, bd), msub(msub(t, ac), bd)};
}
ZS_HD cm31 cmul_m(cm31 x, uint32_t s) { return {mmul(x.a, s), mmul(x.b, s)}; }
ZS_HD cm31 cmul_i(cm31 x) { return {mneg(x.b), x.a}; }
// (a+bi)^-1 = (a - bi) / (a^2 + b^2); a zero norm gives zero like the reference.
ZS_HD cm31 cinv(cm31 x) {
  uint32_t ni = minv(madd(mmul(x.a, x.a), mmul(x.b, x.b)));
  return {mmul(x.a, ni), mmul(mneg(x.b), ni)};
}

struct qm31 {
  cm31 a, b;  // a + b j, j^2 = -i. Wire order: a.a, a.b, b.a, b.b (qm31.zig:91-94)
};
ZS_HD qm31 qzero() { return {{0, 0}, {0, 0}}; }
ZS_HD qm31 qone() { return {{1, 0}, {0, 0}}; }
ZS_HD qm31 qfrom_m31(uint32_t v) { return {{v, 0}, {0, 0}}; }
ZS_HD qm31 qmake(uint32_t w0, uint32_t w1, uint32_t w2, uint32_t w3) { return {{w0, w1}, {w2, w3}}; }
ZS_HD qm31 qadd(qm31 x, qm31 y) { return {cadd(x.a, y.a), cadd(x.b, y.b)}; }
ZS_HD qm31 qsub(qm31 x, qm31 y) { return {csub(x.a, y.a), csub(x.b, y.b)}; }
ZS_HD qm31 qneg(qm31 x) { return {cneg(x.a), cneg(x.b)}; }
// sum_k g_k x_k over QM31 with the four coordinates' products accumulated unreduced in 64 bits:
//   (a + b j)(c + d j) = a c - i b d + (a d + b c) j, and for the words of each factor
//   .a.a: a0 c0 - a1 c1 + b0 d1 + b1 d0    .b.a: a0 d0 - a1 d1 + b0 c0 - b1 c1
//   .a.b: a0 c1 + a1 c0 - b0 d0 + b1 d1    .b.b: a0 d1 + a1 d0 + b0 c1 + b1 c0
// with -v taken as p - v. p 2^32 is a multiple of p, so after every second product a minimum on
// the high word takes it off; then the high word is at most p + 1 and two more products of
// words <= p keep the sum below 2^64. A term is 16 wide multiply-adds and 8 minima, against 9
// reduced products and 27 reduced sums (63 ALU operations) for qmul's Karatsuba form and its sum.
// stacked Rescue 2^18: quotient 230 -> 197 us, DEEP 165 -> 110 us; the linear layer's proof 12.2 ->
// 12.0 ms.
struct QAcc {
  uint64_t v[4] = {0, 0, 0, 0};
  ZS_HD static uint64_t fold(uint64_t x) {
    const uint32_t hi = (uint32_t)(x >> 32);
    return (uint64_t)umin32(hi, hi - P) << 32 | (uint32_t)x;
  }
  ZS_HD static uint64_t two(uint64_t acc, uint32_t a, uint32_t c, uint32_t b, uint32_t d) {
    return fold(acc + (uint64_t)a * c + (uint64_t)b * d);
  }
  ZS_HD void mul_add(const qm31& g, const qm31& x) {
    const uint32_t na1 = P - g.a.b, nb0 = P - g.b.a, nb1 = P - g.b.b;
    v[0] = two(two(v[0], g.a.a, x.a.a, na1, x.a.b), g.b.a, x.b.b, g.b.b, x.b.a);
    v[1] = two(two(v[1], g.a.a, x.a.b, g.a.b, x.a.a), nb0, x.b.a, g.b.b, x.b.b);
    v[2] = two(two(v[2], g.a.a, x.b.a, na1, x.b.b), g.b.a, x.a.a, nb1, x.a.b);
    v[3] = two(two(v[3], g.a.a, x.b.b, g.a.b, x.b.a), g.b.a, x.a.b, g.b.b, x.a.a);
  }
  // 64 -> 31 bits: high word h <= p + 1, so 2^31 m + l with m <= 2p - 1 and l <= p; the sum of
  // m's residue and l is then at most 2p - 1, and one minimum makes it canonical. The last one
  // changes no value; without it the kernels schedule no better (SeededFib 2^12 620 -> 623 us,
  // the other proofs equal).
  ZS_HD static uint32_t canon(uint64_t x) {
    const uint32_t h = (uint32_t)(x >> 32), lo = (uint32_t)x;
    const uint32_t m = umin32(h, h - P) << 1 | lo >> 31;  // h < p now, or 0 or 1 for p and p + 1
    const uint32_t s = umin32(m, m - P) + (lo & P);
    const uint32_t r = umin32(s, s - P);
    return umin32(r, r - P);
  }
  ZS_HD qm31 value() const { return qmake(canon(v[0]), canon(v[1]), canon(v[2]), canon(v[3])); }
};
// qm31.zig:25-33 structure: (ab0 - i ab1, (a+b)(a'+b') - ab0 - ab1).
ZS_HD qm31 qmul(qm31 x, qm31 y) {
#ifdef __CUDA_ARCH__
  QAcc acc;  // the products of one term; 3-way products need fewer multiplies but more ALU work
  acc.mul_add(x, y);
  return acc.value();
#else
  cm31 ab0 = cmul(x.a, y.a), ab1 = cmul(x.b, y.b);
  cm31 cross = cmul(cadd(x.a, x.b), cadd(y.a, y.b));
  return {csub(ab0, cmul_i(ab1)), csub(csub(cross, ab0), ab1)};
#endif
}
ZS_HD qm31 qmul_m(qm31 x, uint32_t s) { return {cmul_m(x.a, s), cmul_m(x.b, s)}; }
// Norm a^2 + i b^2 in CM31; inverse = (a - b j) / norm (qm31.zig:39-48).
ZS_HD cm31 qnorm(qm31 x) { return cadd(cmul(x.a, x.a), cmul_i(cmul(x.b, x.b))); }
ZS_HD qm31 qinv(qm31 x) {
  cm31 ni = cinv(qnorm(x));
  return {cmul(x.a, ni), cmul(cneg(x.b), ni)};
}
ZS_HD qm31 qpow(qm31 x, uint64_t e) {
  qm31 r = qone();
  while (e) {
    if (e & 1) r = qmul(r, x);
    x = qmul(x, x);
    e >>= 1;
  }
  return r;
}
ZS_HD bool qeq(qm31 x, qm31 y) { return x.a.a == y.a.a && x.a.b == y.a.b && x.b.a == y.b.a && x.b.b == y.b.b; }

// qm31.zig:80-83: the primitive 2^32-th root of unity, as LE words.
ZS_HD qm31 q_two_adic_root() { return qmake(0x343d1f60u, 0x6aa03932u, 0x6151d6a0u, 0x3e86e791u); }
ZS_HD qm31 q_root_of_unity(unsigned log_size) {
  return qpow(q_two_adic_root(), (uint64_t)1 << (32 - log_size));
}
// fri.zig:36: FRI_OFFSET = {a = CM31 one, b = CM31 one} = 1 + j.
ZS_HD qm31 q_fri_offset() { return qmake(1, 0, 1, 0); }

// Circle group point over M31 (src/m31/circle/point.zig).
struct cpoint {
  uint32_t x, y;
};
ZS_HD cpoint padd(cpoint p, cpoint q) {
  return {msub(mmul(p.x, q.x), mmul(p.y, q.y)), madd(mmul(p.x, q.y), mmul(p.y, q.x))};
}
ZS_HD cpoint pdbl(cpoint p) { return {msub(mmul(p.x, p.x), mmul(p.y, p.y)), mmul(mmul(p.x, p.y), 2)}; }
ZS_HD cpoint pmul(cpoint p, uint64_t k) {
  cpoint r = {1, 0};
  while (k) {
    if (k & 1) r = padd(r, p);
    p = pdbl(p);
    k >>= 1;
  }
  return r;
}

}  // namespace zs
