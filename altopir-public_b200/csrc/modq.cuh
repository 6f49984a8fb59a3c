// modq.cuh -- exact arithmetic modulo Q = 4294955009 = 2^32 - 12287 on 32-bit residues, shared by host and device.
//
// All inputs are residues in [0, Q) unless stated.  Q > 2^31, so sums overflow 32 bits; the helpers use the wrap of
// unsigned arithmetic, which subtracts 2^32 = Q + 12287, to stay in 32-bit registers.
#pragma once
#include <cstdint>

#if defined(__CUDACC__)
#define ALTO_HD __host__ __device__ __forceinline__
#else
#define ALTO_HD inline
#endif

namespace alto {

constexpr uint32_t kQ32 = 4294955009u;
constexpr uint32_t kFold = 12287u;  // 2^32 mod Q

ALTO_HD uint32_t umin_u32(uint32_t a, uint32_t b) { return a < b ? a : b; }

// (a + b) mod Q.  d = s - Q (mod 2^32).  On a carry the true sum a + b = s + 2^32 >= Q, and d = s + 12287 is that
// sum minus Q.  Without a carry, d < s exactly when s >= Q (below Q the subtraction wraps to s + 12287 > s), so the
// smaller of s and d is the residue.
ALTO_HD uint32_t add_q(uint32_t a, uint32_t b) {
  const uint32_t s = a + b, d = s - kQ32;
  return s < a ? d : umin_u32(s, d);
}

// (a - b) mod Q.
ALTO_HD uint32_t sub_q(uint32_t a, uint32_t b) {
  const uint32_t d = a - b;
  return a < b ? d + kQ32 : d;
}

// x mod Q for any 64-bit x: x = h 2^32 + l = 12287 h + l (mod Q); two folds leave x < 2^32 + 2^28, whose high word
// h is 0 or 1.  With h = 1, x - Q = l + 12287 < Q (l < 2^28); with h = 0 the smaller of l and l - Q (mod 2^32) is the
// residue, as in add_q.
ALTO_HD uint32_t red_q64(uint64_t x) {
  x = (x >> 32) * kFold + (x & 0xffffffffull);
  x = (x >> 32) * kFold + (x & 0xffffffffull);
  const uint32_t t = (uint32_t)x + (uint32_t)(x >> 32) * kFold;
  return umin_u32(t, t - kQ32);
}

// One fold of a 64-bit x: h 2^32 + l -> 12287 h + l, congruent to x mod Q and below 2^46 (not reduced).
ALTO_HD uint64_t fold_q64(uint64_t x) { return (x >> 32) * kFold + (x & 0xffffffffull); }

// (a * b) mod Q for any 32-bit a, b.
ALTO_HD uint32_t mul_q(uint32_t a, uint32_t b) { return red_q64((uint64_t)a * b); }

// Montgomery products: mont_q(a, w 2^32 mod Q) = a w mod Q in [0, Q), for any 32-bit a and w in [0, Q).  With m = lo(x)
// Q^-1 mod 2^32 the low words of x = a w and m Q agree, so (x - m Q) / 2^32 = hi(x) - hi(m Q), above -Q and below Q
// (hi(x) < Q as a < 2^32).  Three multiplications and a conditional add, against four multiplications with their 64-bit
// additions for mul_q, whose operands need no preparation.
constexpr uint32_t inv_mod_2_32(uint32_t a) {  // a^-1 mod 2^32 for odd a: Newton's iteration from a a = 1 (mod 8)
  uint32_t x = a;
  for (int i = 0; i < 4; ++i) x *= 2u - a * x;
  return x;
}
constexpr uint32_t kQInv = inv_mod_2_32(kQ32);
static_assert(kQInv * kQ32 == 1u, "Q^-1 mod 2^32");
ALTO_HD uint32_t mont_q(uint32_t a, uint32_t wm) {
  const uint64_t x = (uint64_t)a * wm;
  const uint32_t hi = (uint32_t)(x >> 32), h = (uint32_t)(((uint64_t)((uint32_t)x * kQInv) * kQ32) >> 32);
  const uint32_t r = hi - h;
  return hi < h ? r + kQ32 : r;
}
ALTO_HD uint32_t to_mont(uint32_t w) { return mul_q(w, kFold); }  // w 2^32 mod Q

// Sums and differences that stay below 2^32 without reaching [0, Q): a any 32-bit representative, b in [0, Q).
// a + b < 2^33 - 12287, so on a carry the low word plus 12287 does not wrap; a - b > -Q, so on a borrow the low word is
// above 12287.  canon_q brings any 32-bit representative into [0, Q).
ALTO_HD uint32_t lazy_add(uint32_t a, uint32_t b) {
  const uint32_t s = a + b;
  return s < a ? s + kFold : s;
}
ALTO_HD uint32_t lazy_sub(uint32_t a, uint32_t b) {
  const uint32_t d = a - b;
  return a < b ? d - kFold : d;
}
ALTO_HD uint32_t canon_q(uint32_t a) { return umin_u32(a, a - kQ32); }

// 2^-l mod Q: (Q + 1) / 2 is the inverse of 2.
ALTO_HD uint32_t inv_pow2_q(int l) {
  uint32_t r = 1;
  for (int i = 0; i < l; ++i) r = mul_q(r, (kQ32 + 1u) / 2u);
  return r;
}

// floor(u / Q) for u < 2^53.  u / 2^32 <= u / Q, so q0 = u >> 32 undershoots; the remainder u - q0 Q =
// (u mod 2^32) + 12287 q0 < 2^32 + 2^35 leaves at most a few more multiples of Q, found the same way.
ALTO_HD uint64_t div_q(uint64_t u) {
  const uint64_t q0 = u >> 32;
  uint64_t r = (u & 0xffffffffull) + q0 * kFold;
  const uint64_t q1 = r >> 32;
  r = (r & 0xffffffffull) + q1 * kFold;
  return q0 + q1 + (r >= kQ32 ? 1u : 0u);
}

// Centred rescale of v in [0, Q) from Q to q1 (q1 < 2^21), rounding half away from zero, result in [0, q1):
// c = v or v - Q (centred), t = trunc((c q1 +- floor(Q/2)) / Q), t + q1 when negative, t - q1 when t = q1
// (src/amx_kernels.cpp:522-529; the reference divides in double precision, which rounds to the same integer).
ALTO_HD uint32_t rescale_q(uint32_t v, uint32_t q1) {
  constexpr uint64_t half = kQ32 / 2u;
  const bool neg = v >= (uint32_t)half;
  const uint32_t mag = neg ? kQ32 - v : v;  // |c| <= ceil(Q / 2)
  // |trunc(x / Q)| = floor((|c| q1 + floor(Q/2)) / Q) <= (q1 + 1) / 2 + 1: below q1 for every q1 >= 2, so a negative
  // c maps to q1 - t (0 for t = 0) and a non-negative one to t
  const uint32_t t = (uint32_t)div_q((uint64_t)mag * q1 + half);
  return neg ? (t ? q1 - t : 0u) : (t >= q1 ? t - q1 : t);
}

}  // namespace alto
