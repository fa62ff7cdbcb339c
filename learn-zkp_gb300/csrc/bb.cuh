// Device arithmetic in BabyBear (p = 15 * 2^27 + 1) and its quintic
// extension E = F[X] / (X^5 - 2) — the field pair of the reference's prime
// benches, Basefold<BabyBear, BinomialExtensionField<BabyBear, 5>, ...>
// (poly-commit/benches/poly-commit.rs:114-123, poly-commit/src/basefold.rs:
// 470-478).
//
// On the device an element is held in Montgomery form a R mod p, R = 2^32:
// a product is one 32 x 32 -> 64 multiply, one low multiply by -p^-1 and one
// multiply-add of p, all on the integer multiplier, plus a conditional
// subtraction.  Values cross the C ABI, the Merkle leaves and the transcript
// in canonical form (bincode of a BabyBear: its canonical value, 4 bytes
// little-endian), converted at those edges.
#pragma once
#include <cstdint>

namespace bb {

constexpr uint32_t P = 2013265921u;        // 0x78000001
constexpr uint32_t P_INV = 0x88000001u;      // p^-1 mod 2^32
constexpr uint32_t R2 = 0x45dddde3u;        // R^2 mod p (to Montgomery form)
constexpr uint32_t MONT_ONE = 0x0ffffffeu;  // R mod p
constexpr uint32_t MONT_INV2 = 0x07ffffffu; // 2^-1 R mod p
constexpr uint32_t W = 2;                   // X^5 = W

__host__ __device__ __forceinline__ uint32_t umin(uint32_t a, uint32_t b) { return a < b ? a : b; }
// a + b mod p for a, b < p: with s = a + b < 2^32, s - p wraps above s
// exactly when s < p, so the smaller of the two is the reduced sum.
__host__ __device__ __forceinline__ uint32_t add(uint32_t a, uint32_t b) {
  const uint32_t s = a + b;
  return umin(s, s - P);
}
// a - b mod p: d = a - b wraps above 2^31 > p when a < b, and then d + p
// wraps back into [0, p).
__host__ __device__ __forceinline__ uint32_t sub(uint32_t a, uint32_t b) {
  const uint32_t d = a - b;
  return umin(d, d + P);
}
// a + b and a - b mod p for a, b < p, left below 2p (2p < 2^32): what mul_shoup, which
// takes any 32-bit word, multiplies next.
__host__ __device__ __forceinline__ uint32_t add_lazy(uint32_t a, uint32_t b) { return a + b; }
__host__ __device__ __forceinline__ uint32_t sub_lazy(uint32_t a, uint32_t b) { return a - b + P; }
// Montgomery product a b R^-1 mod p of a, b < p (R = 2^32): with t = a b and
// m = t p^-1 mod R, m p has the low word of t, so (t - m p) / R is
// hi(t) - hi(m p), in (-p, p); a negative difference wraps and gets p added.
__host__ __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) {
  const uint64_t t = (uint64_t)a * b;
  const uint32_t m = (uint32_t)t * P_INV;
  const uint32_t mh = (uint32_t)(((uint64_t)m * P) >> 32);
  const uint32_t d = (uint32_t)(t >> 32) - mh;
  return umin(d, d + P);
}
// Shoup product a w mod p for any 32-bit a and a fixed w < p, given
// ws = floor(w 2^32 / p): q = hi(a ws) is below a w / p by less than 2, so
// a w - q p (mod 2^32) lies in [0, 2p).  One high multiply instead of the
// Montgomery product's wide and high ones; with a in Montgomery form and w
// canonical, the product stays in Montgomery form.
__host__ __device__ __forceinline__ uint32_t shoup_quot(uint32_t w) { return (uint32_t)(((uint64_t)w << 32) / P); }
#ifdef __CUDACC__
__device__ __forceinline__ uint32_t mul_shoup(uint32_t a, uint2 f) {  // f = (w, shoup_quot(w))
  const uint32_t r = a * f.x - __umulhi(a, f.y) * P;
  return umin(r, r - P);
}
#endif
__host__ __device__ __forceinline__ uint32_t to_mont(uint32_t a) { return mul(a, R2); }
__host__ __device__ __forceinline__ uint32_t from_mont(uint32_t a) { return mul(a, 1u); }

// Extension element: coefficients of 1, X, .., X^4, each in Montgomery form.
struct E5 {
  uint32_t c[5];
};
__host__ __device__ __forceinline__ E5 e_zero() { return E5{{0, 0, 0, 0, 0}}; }
__host__ __device__ __forceinline__ E5 e_from(uint32_t f) { return E5{{f, 0, 0, 0, 0}}; }
__host__ __device__ __forceinline__ E5 e_add(const E5& a, const E5& b) {
  E5 r;
  for (int i = 0; i < 5; ++i) r.c[i] = add(a.c[i], b.c[i]);
  return r;
}
__host__ __device__ __forceinline__ E5 e_sub(const E5& a, const E5& b) {
  E5 r;
  for (int i = 0; i < 5; ++i) r.c[i] = sub(a.c[i], b.c[i]);
  return r;
}
__host__ __device__ __forceinline__ E5 e_scale(const E5& a, uint32_t f) {
  E5 r;
  for (int i = 0; i < 5; ++i) r.c[i] = mul(a.c[i], f);
  return r;
}
// t R^-1 mod p for t < p 2^32 (the Montgomery reduction of a sum of products).
__host__ __device__ __forceinline__ uint32_t reduce(uint64_t t) {
  const uint32_t m = (uint32_t)t * P_INV;
  const uint32_t d = (uint32_t)(t >> 32) - (uint32_t)(((uint64_t)m * P) >> 32);
  return umin(d, d + P);
}
// (sum_i a_i X^i)(sum_j b_j X^j) with X^5 = 2: coefficient k is the sum of the
// five products a_j b_(k-j), those that wrap past X^5 with b doubled.  Four
// products of words below p sum below 2^63.9; the sum is folded to
// hi (2^32 mod p) + lo (below 2^60) before the fifth, so one reduction of less
// than p 2^32 per coefficient replaces one per product.
__host__ __device__ __forceinline__ E5 e_mul(const E5& a, const E5& b) {
  uint32_t bd[5];
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int j = 1; j < 5; ++j) bd[j] = add(b.c[j], b.c[j]);
  E5 r;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
  for (int k = 0; k < 5; ++k) {
    uint64_t s = 0;
#ifdef __CUDA_ARCH__
#pragma unroll
#endif
    for (int j = 0; j < 4; ++j) s += (uint64_t)a.c[j] * (j <= k ? b.c[k - j] : bd[k - j + 5]);
    s = (s >> 32) * MONT_ONE + (uint32_t)s;
    r.c[k] = reduce(s + (uint64_t)a.c[4] * (k == 4 ? b.c[0] : bd[k + 1]));
  }
  return r;
}

}  // namespace bb
