// Device Keccak-f[1600] and the fixed-length Keccak-256 digests of the
// Basefold Merkle trees.
//
// The reference hashes with Plonky3's Keccak256Hash over tiny-keccak 2.0.2
// `Keccak::v256` (original Keccak padding: 0x01 after the message, 0x80 in
// the last byte of the 136-byte rate).  Every message on the hot path fits
// one block: a codeword leaf is one 16-byte field element, a folded-codeword
// leaf is two elements (32 bytes), an inner node is left || right (64 bytes)
// (p3/src/symmetric.rs:11-26, p3/src/merkle_tree.rs:8-21).
//
// Lanes are 64-bit words kept as uint2 (x = low 32 bits); every rotation is
// two funnel shifts.  Constants are FIPS 202's round constants and rho
// offsets (checked against the spec's LFSR and lane walk by the tests).
//
// The Merkle-tree hashes run on bit-interleaved lanes instead: a lane is
// (even bits, odd bits), so a 64-bit rotation by an even amount is two
// 32-bit rotations, by an odd amount two with the halves swapped, and by one
// (theta) a single funnel shift — 6 fewer ALU instructions per round
// (measured on GB300: 4.67 vs 4.51 G permutations/s).  Digests stored in
// the trees stay interleaved, so a node hash reads its children as they are;
// only what leaves the trees (roots to the transcript and the host, query
// paths) is converted back to bytes.
#pragma once
#include <cstdint>

namespace bf {

__constant__ uint2 c_keccak_rc[24] = {
    {0x00000001u, 0x00000000u}, {0x00008082u, 0x00000000u}, {0x0000808au, 0x80000000u},
    {0x80008000u, 0x80000000u}, {0x0000808bu, 0x00000000u}, {0x80000001u, 0x00000000u},
    {0x80008081u, 0x80000000u}, {0x00008009u, 0x80000000u}, {0x0000008au, 0x00000000u},
    {0x00000088u, 0x00000000u}, {0x80008009u, 0x00000000u}, {0x8000000au, 0x00000000u},
    {0x8000808bu, 0x00000000u}, {0x0000008bu, 0x80000000u}, {0x00008089u, 0x80000000u},
    {0x00008003u, 0x80000000u}, {0x00008002u, 0x80000000u}, {0x00000080u, 0x80000000u},
    {0x0000800au, 0x00000000u}, {0x8000000au, 0x80000000u}, {0x80008081u, 0x80000000u},
    {0x00008080u, 0x80000000u}, {0x80000001u, 0x00000000u}, {0x80008008u, 0x80000000u},
};

__device__ __forceinline__ uint2 kx2(uint2 a, uint2 b) { return make_uint2(a.x ^ b.x, a.y ^ b.y); }
__device__ __forceinline__ uint2 kx3(uint2 a, uint2 b, uint2 c) {
  return make_uint2(a.x ^ b.x ^ c.x, a.y ^ b.y ^ c.y);
}
__device__ __forceinline__ uint2 kx5(uint2 a, uint2 b, uint2 c, uint2 d, uint2 e) {
  return make_uint2(a.x ^ b.x ^ c.x ^ d.x ^ e.x, a.y ^ b.y ^ c.y ^ d.y ^ e.y);
}
// a ^ (~b & c)
__device__ __forceinline__ uint2 kchi(uint2 a, uint2 b, uint2 c) {
  return make_uint2(a.x ^ (~b.x & c.x), a.y ^ (~b.y & c.y));
}
// 64-bit rotation by R in two funnel shifts.  (Measured on GB300: funnel
// shifts, LOP3 and IADD3 all issue at half rate on the ALU pipe; a rotation
// rebuilt from integer multiplies needs the quarter-rate IMAD.HI/IMAD.WIDE
// forms and was slower, so rotations stay on the ALU pipe.)
template <int R>
__device__ __forceinline__ uint2 krol(uint2 v) {
  if constexpr (R == 0) {
    return v;
  } else if constexpr (R < 32) {
    return make_uint2(__funnelshift_l(v.y, v.x, R), __funnelshift_l(v.x, v.y, R));
  } else if constexpr (R == 32) {
    return make_uint2(v.y, v.x);
  } else {
    return make_uint2(__funnelshift_l(v.x, v.y, R - 32), __funnelshift_l(v.y, v.x, R - 32));
  }
}

// ---- bit-interleaved lanes --------------------------------------------------
// Even bits of each 32-bit word to its low half, odd bits to its high half
// (an inverse perfect shuffle), and back.
__host__ __device__ __forceinline__ uint32_t bi_unshuffle32(uint32_t x) {
  uint32_t t;
  t = (x ^ (x >> 1)) & 0x22222222u;
  x ^= t ^ (t << 1);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 4)) & 0x00F000F0u;
  x ^= t ^ (t << 4);
  t = (x ^ (x >> 8)) & 0x0000FF00u;
  x ^= t ^ (t << 8);
  return x;
}
__host__ __device__ __forceinline__ uint32_t bi_shuffle32(uint32_t x) {
  uint32_t t;
  t = (x ^ (x >> 8)) & 0x0000FF00u;
  x ^= t ^ (t << 8);
  t = (x ^ (x >> 4)) & 0x00F000F0u;
  x ^= t ^ (t << 4);
  t = (x ^ (x >> 2)) & 0x0C0C0C0Cu;
  x ^= t ^ (t << 2);
  t = (x ^ (x >> 1)) & 0x22222222u;
  x ^= t ^ (t << 1);
  return x;
}
// 64-bit lane (x = low word) -> (even bits, odd bits), and back.
__device__ __forceinline__ uint2 bi_from_lane(uint2 v) {
  const uint32_t lo = bi_unshuffle32(v.x), hi = bi_unshuffle32(v.y);
  return make_uint2(__byte_perm(lo, hi, 0x5410), __byte_perm(lo, hi, 0x7632));
}
__device__ __forceinline__ uint2 bi_to_lane(uint2 v) {
  return make_uint2(bi_shuffle32(__byte_perm(v.x, v.y, 0x5410)), bi_shuffle32(__byte_perm(v.x, v.y, 0x7632)));
}

// FIPS 202 round constants, bit-interleaved (even bits, odd bits).
__constant__ uint2 c_keccak_rc_bi[24] = {
    {0x00000001u, 0x00000000u}, {0x00000000u, 0x00000089u}, {0x00000000u, 0x8000008bu},
    {0x00000000u, 0x80008080u}, {0x00000001u, 0x0000008bu}, {0x00000001u, 0x00008000u},
    {0x00000001u, 0x80008088u}, {0x00000001u, 0x80000082u}, {0x00000000u, 0x0000000bu},
    {0x00000000u, 0x0000000au}, {0x00000001u, 0x00008082u}, {0x00000000u, 0x00008003u},
    {0x00000001u, 0x0000808bu}, {0x00000001u, 0x8000000bu}, {0x00000001u, 0x8000008au},
    {0x00000001u, 0x80000081u}, {0x00000000u, 0x80000081u}, {0x00000000u, 0x80000008u},
    {0x00000000u, 0x00000083u}, {0x00000000u, 0x80008003u}, {0x00000001u, 0x80008088u},
    {0x00000000u, 0x80000088u}, {0x00000001u, 0x00008000u}, {0x00000000u, 0x80008082u},
};

__device__ __forceinline__ uint32_t rotl32(uint32_t x, int k) { return __funnelshift_l(x, x, k); }
// 64-bit rotation by R of an interleaved lane.
template <int R>
__device__ __forceinline__ uint2 krol_bi(uint2 v) {
  if constexpr (R == 0) {
    return v;
  } else if constexpr ((R & 1) == 0) {
    return make_uint2(rotl32(v.x, R / 2), rotl32(v.y, R / 2));
  } else if constexpr (R == 1) {
    return make_uint2(rotl32(v.y, 1), v.x);
  } else {
    return make_uint2(rotl32(v.y, (R + 1) / 2), rotl32(v.x, (R - 1) / 2));
  }
}

template <int R, bool BI>
__device__ __forceinline__ uint2 krot(uint2 v) {
  if constexpr (BI)
    return krol_bi<R>(v);
  else
    return krol<R>(v);
}

// One round: theta, rho and pi into b[], chi back into s[], iota.  BI: the
// lanes are bit-interleaved.
template <bool BI = false>
__device__ __forceinline__ void keccak_round(uint2 s[25], uint2 rc) {
  uint2 C[5], D[5], b[25];
#pragma unroll
  for (int x = 0; x < 5; ++x) C[x] = kx5(s[x], s[x + 5], s[x + 10], s[x + 15], s[x + 20]);
#pragma unroll
  for (int x = 0; x < 5; ++x) D[x] = krot<1, BI>(C[(x + 1) % 5]);
#pragma unroll
  for (int i = 0; i < 25; ++i) s[i] = kx3(s[i], C[(i + 4) % 5], D[i % 5]);
  // b[y + 5 ((2x + 3y) mod 5)] = rot(s[x + 5y], r[x, y])
  b[0] = s[0];
  b[10] = krot<1, BI>(s[1]);
  b[20] = krot<62, BI>(s[2]);
  b[5] = krot<28, BI>(s[3]);
  b[15] = krot<27, BI>(s[4]);
  b[16] = krot<36, BI>(s[5]);
  b[1] = krot<44, BI>(s[6]);
  b[11] = krot<6, BI>(s[7]);
  b[21] = krot<55, BI>(s[8]);
  b[6] = krot<20, BI>(s[9]);
  b[7] = krot<3, BI>(s[10]);
  b[17] = krot<10, BI>(s[11]);
  b[2] = krot<43, BI>(s[12]);
  b[12] = krot<25, BI>(s[13]);
  b[22] = krot<39, BI>(s[14]);
  b[23] = krot<41, BI>(s[15]);
  b[8] = krot<45, BI>(s[16]);
  b[18] = krot<15, BI>(s[17]);
  b[3] = krot<21, BI>(s[18]);
  b[13] = krot<8, BI>(s[19]);
  b[14] = krot<18, BI>(s[20]);
  b[24] = krot<2, BI>(s[21]);
  b[9] = krot<61, BI>(s[22]);
  b[19] = krot<56, BI>(s[23]);
  b[4] = krot<14, BI>(s[24]);
#pragma unroll
  for (int y = 0; y < 25; y += 5) {
#pragma unroll
    for (int x = 0; x < 5; ++x) s[y + x] = kchi(b[y + x], b[y + (x + 1) % 5], b[y + (x + 2) % 5]);
  }
  s[0] = kx2(s[0], rc);
}

// Last round when only the 32-byte digest (lanes 0..3) is wanted: theta is
// still needed in full, but rho/pi/chi only for the five lanes of row y = 0.
template <bool BI = false>
__device__ __forceinline__ void keccak_round_digest(uint2 s[25], uint2 rc) {
  uint2 C[5], D[5];
#pragma unroll
  for (int x = 0; x < 5; ++x) C[x] = kx5(s[x], s[x + 5], s[x + 10], s[x + 15], s[x + 20]);
#pragma unroll
  for (int x = 0; x < 5; ++x) D[x] = krot<1, BI>(C[(x + 1) % 5]);
  // row y = 0 of b takes lanes 0, 6, 12, 18, 24
  const uint2 b0 = kx3(s[0], C[4], D[0]);
  const uint2 b1 = krot<44, BI>(kx3(s[6], C[0], D[1]));
  const uint2 b2 = krot<43, BI>(kx3(s[12], C[1], D[2]));
  const uint2 b3 = krot<21, BI>(kx3(s[18], C[2], D[3]));
  const uint2 b4 = krot<14, BI>(kx3(s[24], C[3], D[4]));
  s[0] = kx2(kchi(b0, b1, b2), rc);
  s[1] = kchi(b1, b2, b3);
  s[2] = kchi(b2, b3, b4);
  s[3] = kchi(b3, b4, b0);
}

template <bool BI>
__device__ __forceinline__ uint2 keccak_rc(int r) {
  return BI ? c_keccak_rc_bi[r] : c_keccak_rc[r];
}

// Full permutation.  The first round is peeled so that the compiler folds
// the lanes a fixed-length message leaves constant (zero or padding).
template <bool BI = false>
__device__ __forceinline__ void keccak_f1600(uint2 s[25]) {
  keccak_round<BI>(s, keccak_rc<BI>(0));
#pragma unroll 2
  for (int r = 1; r < 23; ++r) keccak_round<BI>(s, keccak_rc<BI>(r));
  keccak_round<BI>(s, keccak_rc<BI>(23));
}

// Permutation whose output is only read in lanes 0..3.
template <bool BI = false>
__device__ __forceinline__ void keccak_f1600_digest(uint2 s[25]) {
  keccak_round<BI>(s, keccak_rc<BI>(0));
#pragma unroll 2
  for (int r = 1; r < 23; ++r) keccak_round<BI>(s, keccak_rc<BI>(r));
  keccak_round_digest<BI>(s, keccak_rc<BI>(23));
}

// Absorb `nlanes` message lanes (already in s[0..nlanes)), pad and permute.
// The digest is lanes 0..3 (32 bytes, little-endian).  The padding bits (bit
// 0 of lane nlanes, bit 63 of lane 16) sit at the same word and bit in the
// interleaved form (even bit 0; odd bit 31).
template <bool BI = false>
__device__ __forceinline__ void keccak256_lanes(uint2 s[25], int nlanes) {
#pragma unroll
  for (int i = 0; i < 25; ++i)
    if (i >= nlanes) s[i] = make_uint2(0, 0);
  // nlanes <= 16 here, so the 0x01 byte and the final 0x80 byte never share a lane.
#pragma unroll
  for (int i = 0; i < 17; ++i)
    if (i == nlanes) s[i].x ^= 0x01u;
  s[16].y ^= 0x80000000u;
  keccak_f1600_digest<BI>(s);
}

struct Digest {
  uint4 lo, hi;  // bytes 0..15, 16..31
};

__device__ __forceinline__ Digest digest_from_state(const uint2 s[25]) {
  Digest d;
  d.lo = make_uint4(s[0].x, s[0].y, s[1].x, s[1].y);
  d.hi = make_uint4(s[2].x, s[2].y, s[3].x, s[3].y);
  return d;
}

// ---- Merkle-tree hashes: digests are returned (and stored) interleaved ----

// keccak256 of one 16-byte field element.
__device__ __forceinline__ Digest hash_elem(uint4 e) {
  uint2 s[25];
  s[0] = bi_from_lane(make_uint2(e.x, e.y));
  s[1] = bi_from_lane(make_uint2(e.z, e.w));
  keccak256_lanes<true>(s, 2);
  return digest_from_state(s);
}

// keccak256 of two field elements (32 bytes).
__device__ __forceinline__ Digest hash_pair(uint4 a, uint4 b) {
  uint2 s[25];
  s[0] = bi_from_lane(make_uint2(a.x, a.y));
  s[1] = bi_from_lane(make_uint2(a.z, a.w));
  s[2] = bi_from_lane(make_uint2(b.x, b.y));
  s[3] = bi_from_lane(make_uint2(b.z, b.w));
  keccak256_lanes<true>(s, 4);
  return digest_from_state(s);
}

// keccak256(left || right), 64 bytes, of two interleaved digests: their
// lanes are the message lanes in interleaved form as they are.
__device__ __forceinline__ Digest hash_node(const Digest& l, const Digest& r) {
  uint2 s[25];
  s[0] = make_uint2(l.lo.x, l.lo.y);
  s[1] = make_uint2(l.lo.z, l.lo.w);
  s[2] = make_uint2(l.hi.x, l.hi.y);
  s[3] = make_uint2(l.hi.z, l.hi.w);
  s[4] = make_uint2(r.lo.x, r.lo.y);
  s[5] = make_uint2(r.lo.z, r.lo.w);
  s[6] = make_uint2(r.hi.x, r.hi.y);
  s[7] = make_uint2(r.hi.z, r.hi.w);
  keccak256_lanes<true>(s, 8);
  return digest_from_state(s);
}

// A digest computed on standard lanes, interleaved for storage in a tree.
__device__ __forceinline__ Digest digest_interleaved(const Digest& d) {
  const uint2 l0 = bi_from_lane(make_uint2(d.lo.x, d.lo.y)), l1 = bi_from_lane(make_uint2(d.lo.z, d.lo.w));
  const uint2 l2 = bi_from_lane(make_uint2(d.hi.x, d.hi.y)), l3 = bi_from_lane(make_uint2(d.hi.z, d.hi.w));
  Digest o;
  o.lo = make_uint4(l0.x, l0.y, l1.x, l1.y);
  o.hi = make_uint4(l2.x, l2.y, l3.x, l3.y);
  return o;
}

// An interleaved digest as its 32 bytes (four little-endian lanes).
__device__ __forceinline__ Digest digest_bytes(const Digest& d) {
  const uint2 l0 = bi_to_lane(make_uint2(d.lo.x, d.lo.y)), l1 = bi_to_lane(make_uint2(d.lo.z, d.lo.w));
  const uint2 l2 = bi_to_lane(make_uint2(d.hi.x, d.hi.y)), l3 = bi_to_lane(make_uint2(d.hi.z, d.hi.w));
  Digest o;
  o.lo = make_uint4(l0.x, l0.y, l1.x, l1.y);
  o.hi = make_uint4(l2.x, l2.y, l3.x, l3.y);
  return o;
}

// ---------------------------------------------------------------------------
// Keccak-f[1600] spread over a warp, for latency-bound hashing (the top
// levels of a Merkle tree, the transcript): lane j < 25 holds state word
// A[x][y], j = x + 5y; lanes 25..31 only take part in the shuffles.  A round
// is three dependent shuffle stages: theta's column sum (the other four words
// of the column), theta's neighbour columns, and pi with chi, which reads the
// three rotated words that end up in a row straight from the lanes that
// rotated them.  Measured on GB300 (one block, clock64): 3,920 cycles per
// permutation on one warp per scheduler and 4,250 on two, against 4,680 and
// 5,140 with pi and chi as stages of their own.  A shuffle issues about every
// 4.4 cycles per scheduler, so four warps per scheduler (7,650 cycles) are
// bound by its 18 shuffles per round; a whole permutation on one thread takes
// 8,500 cycles (its 173 instructions per round issue at the half-rate ALU
// pipe's pace) and on a pair of lanes 5,330 (PairKeccak), so a level runs one
// warp per node only while it has at most two nodes per scheduler.
struct WarpKeccak {
  int lane;
  int col[4];            // theta: the other four lanes of this column
  int xm1, xp1;          // theta: lanes of columns x-1, x+1 in this row
  int src0, src1, src2;  // pi and chi: the lanes whose rotated words become B[x], B[x+1], B[x+2] of this row
  int rho;               // rotation of this lane, applied before pi moves the word

  __device__ __forceinline__ WarpKeccak() {
    lane = threadIdx.x & 31;
    const int j = lane < 25 ? lane : 0;
    const int x = j % 5, y = j / 5;
#pragma unroll
    for (int k = 0; k < 4; ++k) col[k] = x + 5 * ((y + 1 + k) % 5);
    xm1 = (x + 4) % 5 + 5 * y;
    xp1 = (x + 1) % 5 + 5 * y;
    // B[X][y] = A[x'][X] with x' = 3 (y - 3X) mod 5 (pi: x = y', y = 2x' + 3y')
    auto pi_lane = [&](int X) { return (3 * ((y - 3 * X) % 5 + 10)) % 5 + 5 * X; };
    src0 = pi_lane(x);
    src1 = pi_lane((x + 1) % 5);
    src2 = pi_lane((x + 2) % 5);
    constexpr int kRho[25] = {0,  1,  62, 28, 27, 36, 44, 6,  55, 20, 3,  10, 43,
                              25, 39, 41, 45, 15, 21, 8,  18, 2,  61, 56, 14};
    int r = 0;
#pragma unroll
    for (int k = 0; k < 25; ++k)
      if (k == j) r = kRho[k];
    rho = r;
  }

  static __device__ __forceinline__ uint2 shfl(uint2 v, int src) {
    return make_uint2(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
  }

  // All 32 lanes call this; `a` is this lane's word (interleaved when BI).
  template <bool BI>
  __device__ __forceinline__ uint2 permute(uint2 a) const {
    // the lane's rotation: swap the halves or not, then a 32-bit (BI) or a
    // funnel shift per half
    const bool swap = BI ? (rho & 1) != 0 : (rho & 32) != 0;
    const int k0 = BI ? (rho + 1) >> 1 : rho & 31, k1 = BI ? rho >> 1 : rho & 31;
#pragma unroll 4
    for (int r = 0; r < 24; ++r) {
      uint2 rc = keccak_rc<BI>(r);
      if (lane != 0) rc = make_uint2(0, 0);
      const uint2 c1 = shfl(a, col[0]), c2 = shfl(a, col[1]), c3 = shfl(a, col[2]), c4 = shfl(a, col[3]);
      const uint2 c = kx5(a, c1, c2, c3, c4);  // C[x]
      const uint2 cm = shfl(c, xm1), cp = shfl(c, xp1);
      const uint2 t = kx3(a, cm, krot<1, BI>(cp));  // theta
      const uint32_t u = swap ? t.y : t.x, v = swap ? t.x : t.y;
      const uint2 q = BI ? make_uint2(rotl32(u, k0), rotl32(v, k1))
                         : make_uint2(__funnelshift_l(v, u, k0), __funnelshift_l(u, v, k1));  // rho
      const uint2 b0 = shfl(q, src0), b1 = shfl(q, src1), b2 = shfl(q, src2);  // pi, chi's row
      a = kx2(kchi(b0, b1, b2), rc);                                           // chi, iota
    }
    return a;
  }
};

// Interleaved Keccak-f[1600] on a pair of lanes: the even lane holds the even
// bits of all 25 words, the odd lane the odd bits (s[i], 32 bits).  Only theta's
// rotation by one and the odd rotations of rho cross between them (18 shuffles
// per round); the rest is half of a one-thread permutation's work per lane.
// Measured on GB300: 5,330 cycles per permutation on one warp per scheduler
// (16 states per warp) against 8,500 for one thread per state, 9,290 on two
// warps per scheduler, so it serves levels of 9 to 64 nodes per block.
struct PairKeccak {
  bool odd;
  __device__ __forceinline__ PairKeccak() { odd = (threadIdx.x & 1u) != 0; }

  template <int R>
  __device__ __forceinline__ uint32_t rot(uint32_t v) const {
    if constexpr (R == 0) {
      return v;
    } else if constexpr ((R & 1) == 0) {
      return rotl32(v, R / 2);
    } else {  // even bits take rotl(odd bits, (R + 1) / 2), odd bits rotl(even bits, (R - 1) / 2)
      const uint32_t o = __shfl_xor_sync(0xffffffffu, v, 1);
      return __funnelshift_l(o, o, odd ? (R - 1) / 2 : (R + 1) / 2);
    }
  }

  __device__ __forceinline__ void round(uint32_t s[25], int r) const {
    const uint2 rc = c_keccak_rc_bi[r];
    uint32_t C[5], D[5], b[25];
#pragma unroll
    for (int x = 0; x < 5; ++x) C[x] = s[x] ^ s[x + 5] ^ s[x + 10] ^ s[x + 15] ^ s[x + 20];
#pragma unroll
    for (int x = 0; x < 5; ++x) D[x] = rot<1>(C[(x + 1) % 5]);
#pragma unroll
    for (int i = 0; i < 25; ++i) s[i] ^= C[(i + 4) % 5] ^ D[i % 5];
    b[0] = s[0];
    b[10] = rot<1>(s[1]);
    b[20] = rot<62>(s[2]);
    b[5] = rot<28>(s[3]);
    b[15] = rot<27>(s[4]);
    b[16] = rot<36>(s[5]);
    b[1] = rot<44>(s[6]);
    b[11] = rot<6>(s[7]);
    b[21] = rot<55>(s[8]);
    b[6] = rot<20>(s[9]);
    b[7] = rot<3>(s[10]);
    b[17] = rot<10>(s[11]);
    b[2] = rot<43>(s[12]);
    b[12] = rot<25>(s[13]);
    b[22] = rot<39>(s[14]);
    b[23] = rot<41>(s[15]);
    b[8] = rot<45>(s[16]);
    b[18] = rot<15>(s[17]);
    b[3] = rot<21>(s[18]);
    b[13] = rot<8>(s[19]);
    b[14] = rot<18>(s[20]);
    b[24] = rot<2>(s[21]);
    b[9] = rot<61>(s[22]);
    b[19] = rot<56>(s[23]);
    b[4] = rot<14>(s[24]);
#pragma unroll
    for (int y = 0; y < 25; y += 5) {
#pragma unroll
      for (int x = 0; x < 5; ++x) s[y + x] = b[y + x] ^ (~b[y + (x + 1) % 5] & b[y + (x + 2) % 5]);
    }
    s[0] ^= odd ? rc.y : rc.x;
  }

  // Pads the `nlanes` message lanes in s[0 .. nlanes) and permutes; the
  // digest is s[0 .. 4).  All 32 lanes of the warp call this.
  __device__ __forceinline__ void keccak256(uint32_t s[25], int nlanes) const {
#pragma unroll
    for (int i = 0; i < 25; ++i)
      if (i >= nlanes) s[i] = 0;
#pragma unroll
    for (int i = 0; i < 17; ++i)
      if (i == nlanes && !odd) s[i] ^= 0x01u;  // bit 0 of the lane after the message
    if (odd) s[16] ^= 0x80000000u;             // bit 63 of lane 16
    round(s, 0);
#pragma unroll 2
    for (int r = 1; r < 24; ++r) round(s, r);
  }
};

// ---- a block's part of a Merkle tree ----------------------------------------
// A digest in shared memory is eight words (uint2 per state lane: even bits,
// odd bits); a block keeps the level it just made there, since reading it
// back from global memory would add an L2 round trip to every level.
constexpr int kTreeThreads = 256;  // threads of a block that runs tree levels
constexpr int kTreeWarps = kTreeThreads / 32;
constexpr int kTreeBlockLog = 9;   // at most 2^9 leaves per block
struct TreeShared {
  uint4 a[2 << (kTreeBlockLog - 1)];  // 2^8 digests
  uint4 b[2 << (kTreeBlockLog - 2)];  // 2^7 digests
};

// One level: hash t < cnt (a power of two) goes to dst_s (shared, packed) and
// dst_g (global, digest t at dst_g + 2 t gstride).  A node's message (LANES 8)
// is the digests t and t + cnt of `src` (digest t at src + 2 t stride); a
// leaf's (LANES < 8) is the LANES interleaved lanes at (const uint2*)src +
// LANES t.  All threads of a block of kTreeThreads call this; the caller
// synchronizes around it.  The form per count is the measured fastest (see
// WarpKeccak and PairKeccak): one warp per hash up to 8, a pair of lanes up to
// 64, one thread above.
template <int LANES>
__device__ __forceinline__ void hash_level_block(const WarpKeccak& wk, const uint4* src, size_t stride, uint32_t cnt,
                                                 uint4* dst_s, uint4* dst_g, size_t gstride) {
  constexpr bool NODE = LANES == 8;
  auto first = [&](uint32_t t) {  // the lanes of the message, or of a node's left child
    return NODE ? reinterpret_cast<const uint2*>(src + 2 * stride * t)
                : reinterpret_cast<const uint2*>(src) + LANES * (size_t)t;
  };
  auto second = [&](uint32_t t) { return reinterpret_cast<const uint2*>(src + 2 * stride * (t + cnt)); };
  if (cnt <= (uint32_t)kTreeWarps) {
    const uint32_t t = threadIdx.x >> 5;
    if (t >= cnt) return;
    uint2 a = make_uint2(0, 0);
    if (wk.lane < (NODE ? 4 : LANES)) a = first(t)[wk.lane];
    else if (NODE && wk.lane < 8) a = second(t)[wk.lane - 4];
    if (wk.lane == LANES) a.x ^= 0x01u;     // pad10*1 after the message
    if (wk.lane == 16) a.y ^= 0x80000000u;  // last byte of the 136-byte rate
    a = wk.permute<true>(a);
    if (wk.lane < 4) {
      reinterpret_cast<uint2*>(dst_s + 2 * t)[wk.lane] = a;
      reinterpret_cast<uint2*>(dst_g + 2 * gstride * t)[wk.lane] = a;
    }
  } else if (cnt <= 64) {
    if ((threadIdx.x & ~31u) >= 2 * cnt) return;  // whole warps: cnt is a multiple of 16
    const PairKeccak pk;
    const uint32_t t = threadIdx.x >> 1, h = threadIdx.x & 1u;
    const uint32_t* l = reinterpret_cast<const uint32_t*>(first(t)) + h;
    uint32_t s[25];
#pragma unroll
    for (int i = 0; i < (NODE ? 4 : LANES); ++i) s[i] = l[2 * i];
    if (NODE) {
      const uint32_t* r = reinterpret_cast<const uint32_t*>(second(t)) + h;
#pragma unroll
      for (int i = 0; i < 4; ++i) s[4 + i] = r[2 * i];
    }
    pk.keccak256(s, LANES);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      reinterpret_cast<uint32_t*>(dst_s + 2 * t)[2 * i + h] = s[i];
      reinterpret_cast<uint32_t*>(dst_g + 2 * gstride * t)[2 * i + h] = s[i];
    }
  } else {
    for (uint32_t t = threadIdx.x; t < cnt; t += kTreeThreads) {
      uint2 s[25];
      const uint2* l = first(t);
#pragma unroll
      for (int i = 0; i < (NODE ? 4 : LANES); ++i) s[i] = l[i];
      if (NODE) {
        const uint2* r = second(t);
#pragma unroll
        for (int i = 0; i < 4; ++i) s[4 + i] = r[i];
      }
      keccak256_lanes<true>(s, LANES);
      const Digest d = digest_from_state(s);
      dst_s[2 * t] = d.lo;
      dst_s[2 * t + 1] = d.hi;
      dst_g[2 * gstride * t] = d.lo;
      dst_g[2 * gstride * t + 1] = d.hi;
    }
  }
}

// Levels 1 .. k (k <= kTreeBlockLog) above 2^k digests at `src` (digest t at
// src + 2 t stride), the block's share b of a tree level of n nodes: node t of
// level j is node b + t (n >> k) of that level, and the levels lie one after
// another from `out`.  Odd levels pass through o0, even ones through o1
// (shared; 2^(k-1) and 2^(k-2) digests).  Returns where the level-k digest is
// (src when k = 0).  All threads of a block of kTreeThreads call this; it ends
// synchronized.
__device__ __forceinline__ const uint4* tree_block(const WarpKeccak& wk, uint4* o0, uint4* o1, const uint4* src,
                                                   size_t stride, uint4* out, size_t n, size_t b, int k) {
  const size_t nk = n >> k;
  for (int j = 1; j <= k; ++j) {
    uint4* o = (j & 1) ? o0 : o1;
    hash_level_block<8>(wk, src, stride, 1u << (k - j), o, out + 2 * b, nk);
    __syncthreads();
    src = o;
    stride = 1;
    n >>= 1;
    out += 2 * n;
  }
  return src;
}

// keccak256 of matrix rows of `words` 32-bit words (`base`, row after row), one
// lane per row, the 32 rows [r0, r0 + 32) per warp.  The 136-byte rate is 34
// words, so every block of every row starts on a word: the warp copies a block of
// its rows into shared memory (`st`: two stages of kStageWords words, 16-byte
// aligned) while it permutes the block before, with asynchronous copies whose lanes
// read whole row runs, 8 bytes each where rows are an even number of words; then each lane
// absorbs its row, conv applied to every word.  The 0x01 pad word follows the
// message and 0x80 ends the last block.  The row is absorbed and permuted on
// plain lanes (interleaving 17 message lanes per block would cost more than the
// interleaved rounds save); only the four digest lanes are interleaved, the
// trees' form.  Bound by the ALU pipe: the permutations alone
// take 85 to 95% of the time.  Measured on GB300 before, with loads through
// registers, padding computed for every word and no copy ahead of its use: 2^20
// rows of 256 words 2122 us and now 1901, 2^17 rows of 1024 words 1047 and 941,
// 2^15 rows of 2048 words 684 and 541.
constexpr int kRateWords = 34;  // a stage's row pitch too: lane r's 8-byte words at 34 r meet no bank twice
constexpr int kStageWords = 32 * kRateWords;
__device__ __forceinline__ void copy_async8(uint32_t* dst, const uint32_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
__device__ __forceinline__ void copy_async4(uint32_t* dst, const uint32_t* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
               : "memory");
}
// The words [34 blk, 34 blk + 34) of the warp's rows, as far as they exist.
__device__ __forceinline__ void stage_rows(uint32_t* st, const uint32_t* __restrict__ base, size_t r0, size_t rows,
                                           uint32_t words, uint32_t blk) {
  const uint32_t lane = threadIdx.x & 31u, c0 = blk * kRateWords;
  const uint32_t n = words - c0 < (uint32_t)kRateWords ? words - c0 : (uint32_t)kRateWords;
  const uint32_t in = rows - r0 < 32 ? (uint32_t)(rows - r0) : 32u;  // rows there are
  const uint32_t* tile = base + r0 * words + c0;
  if ((words & 1u) == 0) {  // 16 lanes a row, then the last 8 bytes with a lane per row
    const uint32_t h = lane >> 4, c = 2 * (lane & 15u);
    const uint32_t* src = tile + (size_t)h * words + c;
    uint32_t* dst = st + h * kRateWords + c;
    const uint32_t have = c < n && h < in ? (in - h + 1) / 2 : 0;  // this lane's rows
    if (have == 16) {
#pragma unroll
      for (int k = 0; k < 16; ++k, src += 2 * (size_t)words) copy_async8(dst + 2 * k * kRateWords, src);
    } else {
      for (uint32_t k = 0; k < have; ++k) copy_async8(dst + 2 * k * kRateWords, src + 2 * (size_t)k * words);
    }
    if (n > 32 && lane < in) copy_async8(st + lane * kRateWords + 32, tile + (size_t)lane * words + 32);
  } else {  // a row per instruction, then the last two words with a lane per row
    if (lane < n)
      for (uint32_t k = 0; k < in; ++k) copy_async4(st + k * kRateWords + lane, tile + (size_t)k * words + lane);
    for (uint32_t i = 32; i < n; ++i)
      if (lane < in) copy_async4(st + lane * kRateWords + i, tile + (size_t)lane * words + i);
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
template <class Conv>
__device__ __forceinline__ Digest keccak_rows_warp(uint32_t* st, const uint32_t* __restrict__ base, size_t r0,
                                                   size_t rows, uint32_t words, const Conv& conv) {
  const uint32_t lane = threadIdx.x & 31u;
  uint2 s[25];
#pragma unroll
  for (int i = 0; i < 25; ++i) s[i] = make_uint2(0, 0);
  const uint32_t last = words / kRateWords;
  stage_rows(st, base, r0, rows, words, 0);
  for (uint32_t blk = 0;; ++blk) {
    const uint2* row = reinterpret_cast<const uint2*>(st + (blk & 1u) * kStageWords + lane * kRateWords);
    if (blk < last) {
      stage_rows(st + (~blk & 1u) * kStageWords, base, r0, rows, words, blk + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      __syncwarp();
#pragma unroll
      for (int k = 0; k < 17; ++k) {
        const uint2 v = row[k];
        s[k].x ^= conv(v.x);
        s[k].y ^= conv(v.y);
      }
      __syncwarp();  // the stage may be refilled
      keccak_f1600<false>(s);
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncwarp();
      const int n = (int)(words - last * kRateWords);
      auto pad = [&](int i, uint32_t v) { return (i < n ? conv(v) : i == n ? 0x01u : 0u) ^ (i == 33 ? 0x80000000u : 0u); };
#pragma unroll
      for (int k = 0; k < 17; ++k) {
        const uint2 v = row[k];
        s[k].x ^= pad(2 * k, v.x);
        s[k].y ^= pad(2 * k + 1, v.y);
      }
      __syncwarp();
      keccak_f1600_digest<false>(s);
      break;
    }
  }
#pragma unroll
  for (int i = 0; i < 4; ++i) s[i] = bi_from_lane(s[i]);
  return digest_from_state(s);
}

__device__ __forceinline__ Digest load_digest(const uint4* p, size_t i) {
  Digest d;
  d.lo = p[2 * i];
  d.hi = p[2 * i + 1];
  return d;
}
__device__ __forceinline__ void store_digest(uint4* p, size_t i, const Digest& d) {
  p[2 * i] = d.lo;
  p[2 * i + 1] = d.hi;
}

}  // namespace bf
