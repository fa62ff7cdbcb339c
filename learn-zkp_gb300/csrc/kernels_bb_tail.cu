// The prime-field open's transcript on the device and its last rounds.
//
//  * bb_transcript_round_kernel: the transcript step of one large round
//    (basefold.rs:340-362 with sumcheck/src/lib.rs:81-103 and EvalImprProver's
//    round polynomial, eval_impr.rs:41-58, 150-162); the fold and fix kernels
//    of the round read the challenge from device memory.
//  * bb_tail_kernel: every remaining round once a fold has at most kBbTailMax
//    outputs — fold, leaves, Merkle levels, fix with the next round's sums and
//    the transcript step — in one block.
#include <cuda_runtime.h>

#include <cstdint>

#include "bb.cuh"
#include "bb_internal.h"
#include "bf_internal.h"
#include "keccak.cuh"
#include "launch.cuh"

namespace bf {

using bb::E5;

namespace {

// ---- extension arithmetic by one warp ---------------------------------------
// Lanes 5 g .. 5 g + 4 (g < 6) hold the five coefficients of an element, so a
// warp multiplies up to six pairs at once: lane 5 g + k gathers the five products
// of coefficient k with ten shuffles and reduces once.
struct ELane {
  int base, k;  // first lane of this lane's group, coefficient of this lane
  __device__ __forceinline__ ELane() {
    const int lane = threadIdx.x & 31;
    base = lane - lane % 5;
    k = lane % 5;
  }
  __device__ __forceinline__ int group() const { return base / 5; }
  __device__ __forceinline__ uint32_t one() const { return k == 0 ? bb::MONT_ONE : 0u; }
  // the coefficients of the element in group g, in every group
  __device__ __forceinline__ uint32_t from(uint32_t v, int g) const { return __shfl_sync(0xffffffffu, v, 5 * g + k); }
  // the product (bb::e_mul's sums, one coefficient per lane)
  __device__ __forceinline__ uint32_t mul(uint32_t a, uint32_t b) const {
    uint64_t s = 0;
#pragma unroll
    for (int j = 0; j < 5; ++j) {
      const uint32_t aj = __shfl_sync(0xffffffffu, a, base + j);
      uint32_t bj = __shfl_sync(0xffffffffu, b, base + (k - j + (j > k ? 5 : 0)));
      if (j > k) bj = bb::add(bj, bj);
      if (j == 4) s = (s >> 32) * bb::MONT_ONE + (uint32_t)s;
      s += (uint64_t)aj * bj;
    }
    return bb::reduce(s);
  }
};

// ---- the transcript step, one warp --------------------------------------------
// Shared memory of the step: the transcript and the round's message (root, then
// the compressed round polynomial, canonical words).
struct BbStepShared {
  BbTranscript t;
  uint32_t msg[18];
};

// keccak256's last block: the first `len` < 136 bytes at `p` (8-byte aligned)
// as this lane's message word, padded.
__device__ __forceinline__ uint2 padded_word(const WarpKeccak& wk, const uint8_t* p, int len) {
  uint2 w = make_uint2(0, 0);
  if (wk.lane < 17) {
    const int n = len - 8 * wk.lane;  // message bytes from this word on
    if (n > 0) w = reinterpret_cast<const uint2*>(p)[wk.lane];
    if (n >= 0 && n < 8) {  // cut after n bytes, then the 0x01 byte
      const uint64_t keep = ((uint64_t)1 << (8 * n)) - 1;
      const uint64_t v = ((((uint64_t)w.y << 32) | w.x) & keep) | ((uint64_t)1 << (8 * n));
      w = make_uint2((uint32_t)v, (uint32_t)(v >> 32));
    }
    if (wk.lane == 16) w.y ^= 0x80000000u;
  }
  return w;
}

// The step in three parts, each by one warp, so that only the challenge stands
// between a round's root and its fold.  From the tree's end to the step's end it
// measured 4.0 us on GB300, 5.3 with all three after the root, 20.9 with one lane
// doing the products one after another, the delta factor rebuilt from all challenges
// and the challenge popped byte by byte.
//
// bb_message: the round polynomial from S, this lane's coefficient of the round's
// sum (Montgomery, the same in every group).
__device__ __forceinline__ void bb_message(BbStepShared& sh, const BbRoundConsts* c, int ri, uint32_t S) {
  const ELane el;
  const int lane = threadIdx.x & 31, k = el.k, g = el.group();
  BbTranscript& t = sh.t;
  const uint32_t cf = __ldcg(&c->cf[ri].c[k]), rinv = __ldcg(&c->r_inv[ri].c[k]), r = __ldcg(&c->r[ri].c[k]);
  const uint32_t omr = bb::sub(el.one(), r);
  const uint32_t claim = t.claim.c[k], delta = t.delta.c[k];
  // c0 = cf S, c1 = (claim - (1 - r) c0) / r - c0; the round polynomial is
  // (c0 + c1 X)(d0 + d1 X) with d0 = delta (1 - r), d1 = delta (2 r - 1)
  const uint32_t m1 = el.mul(g == 0 ? cf : delta, g == 0 ? S : g == 1 ? omr : bb::sub(r, omr));
  const uint32_t c0 = el.from(m1, 0), d0 = el.from(m1, 1), d1 = el.from(m1, 2);
  const uint32_t m2 = el.mul(c0, g == 0 ? omr : d0);
  const uint32_t rp0 = el.from(m2, 1);
  const uint32_t c1 = bb::sub(el.mul(bb::sub(claim, el.from(m2, 0)), rinv), c0);
  const uint32_t rp2 = el.mul(c1, d1);
  if (lane < 5) {
    sh.msg[8 + lane] = bb::from_mont(rp0);  // Eval::compress_round_poly keeps c0 and c2
    t.c0.c[k] = c0;
    t.c1.c[k] = c1;
    t.r.c[k] = r;
  } else if (lane < 10) {
    sh.msg[13 + k] = bb::from_mont(rp2);
  }
  __syncwarp();
}

// bb_claim: EvalProver's claim c0 + c1 x (eval.rs:108-111) and the next delta:
// delta (2 r x + 1 - r - x) (multilinear.rs:224-229).
__device__ __forceinline__ void bb_claim(BbStepShared& sh) {
  const ELane el;
  const int lane = threadIdx.x & 31, k = el.k, g = el.group();
  BbTranscript& t = sh.t;
  const uint32_t r = t.r.c[k], x = t.x.c[k], c0 = t.c0.c[k], delta = t.delta.c[k];
  const uint32_t m = el.mul(g == 0 ? t.c1.c[k] : r, x);
  const uint32_t rx = el.from(m, 1);
  const uint32_t f = bb::sub(bb::sub(bb::add(bb::add(rx, rx), el.one()), r), x);
  const uint32_t nd = el.mul(delta, f);
  __syncwarp();
  if (lane < 5) {
    t.claim.c[k] = bb::add(c0, m);
    t.delta.c[k] = nd;
  }
  __syncwarp();
}

// bb_challenge: observes the root and the message, samples t.x.
__device__ __forceinline__ void bb_challenge(const WarpKeccak& wk, BbStepShared& sh, const uint4* root, uint8_t* rec) {
  const ELane el;
  const int lane = wk.lane, k = el.k;
  BbTranscript& t = sh.t;
  if (lane >= 28) {  // the root's 32 bytes
    const uint2 v = bi_to_lane(reinterpret_cast<const uint2*>(root)[lane - 28]);
    sh.msg[2 * (lane - 28)] = v.x;
    sh.msg[2 * (lane - 28) + 1] = v.y;
  }
  __syncwarp();
  // observe the root and the polynomial (challenger.rs:51-60): appended to the
  // pending input, whole blocks absorbed, the output cleared
  uint2 a = lane < 25 ? t.A[lane] : make_uint2(0, 0);
  int len = (int)t.pend_len;
  if (lane < 18) {
    const uint32_t w = sh.msg[lane];
    reinterpret_cast<uint32_t*>(rec)[lane] = w;
    if ((len & 3) == 0) {
      *reinterpret_cast<uint32_t*>(t.pend + len + 4 * lane) = w;
    } else {
#pragma unroll
      for (int b = 0; b < 4; ++b) t.pend[len + 4 * lane + b] = (uint8_t)(w >> (8 * b));
    }
  }
  __syncwarp();
  len += 72;  // at most 135 + 72: one block at most
  if (len >= 136) {
    if (lane < 17) a = kx2(a, reinterpret_cast<const uint2*>(t.pend)[lane]);
    a = wk.permute<false>(a);
    len -= 136;
    uint8_t keep[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) keep[q] = lane + 32 * q < len ? t.pend[136 + lane + 32 * q] : 0;
    __syncwarp();
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (lane + 32 * q < len) t.pend[lane + 32 * q] = keep[q];
    __syncwarp();
  }
  // sample (challenger.rs:62-74): the digest of the input becomes the output and
  // the new input; a BabyBear is 4 bytes popped from the end, little-endian, shifted
  // right by one, redrawn while >= p
  a = wk.permute<false>(kx2(a, padded_word(wk, t.pend, len)));
  uint32_t x = 0;
  int got = 0, used = 0;
  for (;;) {
    const int wi = (7 - lane) & 7;  // lane j < 8 holds the j-th word popped
    const uint32_t wx = __shfl_sync(0xffffffffu, a.x, wi >> 1), wy = __shfl_sync(0xffffffffu, a.y, wi >> 1);
    const uint32_t v = __byte_perm((wi & 1) ? wy : wx, 0, 0x0123) >> 1;
    uint32_t ok = __ballot_sync(0xffffffffu, lane < 8 && v < bb::P);
    while (ok && got < 5) {
      const int j = __ffs(ok) - 1;
      ok &= ok - 1;
      const uint32_t xv = __shfl_sync(0xffffffffu, v, j);
      if (k == got) x = bb::to_mont(xv);
      ++got;
      used = j + 1;
    }
    if (got == 5) break;
    if (lane >= 4) a = make_uint2(0, 0);  // the output is used up: the digest of the digest
    if (lane == 4) a.x = 0x01u;
    if (lane == 16) a.y = 0x80000000u;
    a = wk.permute<false>(a);
  }
  if (lane < 5) t.x.c[k] = x;
  if (lane < 4) {
    reinterpret_cast<uint2*>(t.pend)[lane] = a;
    reinterpret_cast<uint2*>(t.out)[lane] = a;
  }
  if (lane < 25) t.A[lane] = make_uint2(0, 0);  // the digest is the whole new input, still pending
  if (lane == 0) {
    t.pend_len = 32;
    t.out_len = (uint32_t)(32 - 4 * used);
  }
  __syncwarp();
}

constexpr int kTrWords = (int)(sizeof(BbTranscript) / sizeof(uint2));
__device__ __forceinline__ void tr_copy(BbTranscript* dst, const BbTranscript* src) {
  for (int q = threadIdx.x; q < kTrWords; q += blockDim.x)
    reinterpret_cast<uint2*>(dst)[q] = reinterpret_cast<const uint2*>(src)[q];
}
__device__ __forceinline__ void tr_load(BbTranscript* dst, const BbTranscript* src) {  // past L1
  for (int q = threadIdx.x; q < kTrWords; q += blockDim.x)
    reinterpret_cast<uint2*>(dst)[q] = __ldcg(reinterpret_cast<const uint2*>(src) + q);
}

__device__ __forceinline__ E5 ld_e5(const uint32_t* p, size_t i) {
  E5 e;
#pragma unroll
  for (int k = 0; k < 5; ++k) e.c[k] = p[5 * i + k];
  return e;
}
__device__ __forceinline__ void st_e5(uint32_t* p, size_t i, const E5& e) {
#pragma unroll
  for (int k = 0; k < 5; ++k) p[5 * i + k] = e.c[k];
}

}  // namespace

// early: the launch before this one is a tree's, and a block of this grid starts
// only after every block of that one has waited for all launches before it, among
// them the ones that wrote the transcript and the sums: those are read (past L1) and
// the message is made before the wait, which is left for the root alone (the rules:
// launch.cuh).
__global__ void __launch_bounds__(32) bb_transcript_round_kernel(BbTranscript* t, const BbRoundConsts* c, int ri,
                                                                const uint4* root_dev, unsigned long long* sums,
                                                                int canonical, uint32_t* x_out, uint8_t* rec,
                                                                bool first, bool early) {
  __shared__ BbStepShared sh;
  const WarpKeccak wk;
  if (!early) chain_wait();
  tr_load(&sh.t, t);
  const uint32_t v = (uint32_t)(__ldcg(sums + threadIdx.x % 5) % bb::P);
  __syncwarp();
  if (!first) bb_claim(sh);
  bb_message(sh, c, ri, canonical ? bb::to_mont(v) : v);
  if (early) chain_wait();
  if (threadIdx.x < 5) sums[threadIdx.x] = 0;  // for the fix that adds up the next round's
  bb_challenge(wk, sh, root_dev, rec);
  if (threadIdx.x < 5) x_out[threadIdx.x] = sh.t.x.c[threadIdx.x];
  tr_copy(t, &sh.t);
}

// The last rounds in one block of eight warps, everything but the outputs in
// shared memory.  While warp 0 samples the challenge the others interpolate:
// l = (lo + hi) / 2 and h - l with h = (lo - hi) t need no challenge, so a fold
// output is one product after it.  The claim and the next round's message are made
// while the leaves are hashed, by a warp that has no hash there.  Each level of
// hashes runs in the form that is fastest for its count (hash_level_block).  Bound by
// the chain of dependent permutations (one per level, leaf and challenge); a round
// took a launch each for fold, fix, sums, transcript and two for the tree before.
// Measured on GB300: 127 us for the last eight rounds of a 2^13 x 5 open (131 with
// claim and message between root and challenge), whose commit, evaluation and open
// took 1,127 us with a launch per step and 916 with this kernel alone.
__global__ void __launch_bounds__(kTreeThreads, 1) bb_tail_kernel(BbTail p) {
  __shared__ BbStepShared sh;
  __shared__ uint32_t pi_a[2 * kBbTailMax * 5], pi_b[kBbTailMax * 5];  // l, then h - l of a fold's input
  __shared__ uint32_t poly[kBbTailMax * 5];                            // the sumcheck polynomial after each fix
  __shared__ __align__(16) uint2 msg[kBbTailMax / 2 * 5];              // leaf messages, interleaved lanes
  __shared__ TreeShared ts;
  __shared__ unsigned long long sums[2][5];  // this round's sum and the next one's
  const WarpKeccak wk;
  const int warp = threadIdx.x >> 5;
  if (!p.early) chain_wait();
  tr_load(&sh.t, p.t);
  if (threadIdx.x < 10) sums[threadIdx.x / 5][threadIdx.x % 5] = 0;
  __syncthreads();
  // sum over the block of h[b] v for the thread's b, into acc (Montgomery sums)
  auto add_sums = [&](const E5& part, unsigned long long* acc) {
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      uint32_t v = part.c[q];
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) v = bb::add(v, __shfl_xor_sync(0xffffffffu, v, o));
      if (wk.lane == 0 && v) atomicAdd(acc + q, (unsigned long long)v);
    }
  };
  auto ld_poly = [&](size_t b) {  // the polynomial before the first fix
    if (p.poly_base) return bb::e_from(bb::to_mont(p.poly[b]));
    E5 e;
#pragma unroll
    for (int q = 0; q < 5; ++q) e.c[q] = __ldcg(p.poly + 5 * b + q);
    return e;
  };
  {  // round i0's sum, as early as the transcript round's
    const size_t n = (size_t)1 << (p.i0 + p.lk);
    E5 part = bb::e_zero();
    for (size_t b = threadIdx.x; b < n; b += kTreeThreads)
      part = bb::e_add(part, bb::e_mul(ld_e5(p.heq, b), ld_poly(b)));
    add_sums(part, sums[0]);
  }
  __syncthreads();
  if (warp == 0) {
    if (!p.first) bb_claim(sh);
    bb_message(sh, p.c, p.i0 + p.lk, (uint32_t)(sums[0][wk.lane % 5] % bb::P));
  }
  if (p.early) chain_wait();
  __syncthreads();
  const uint4* root = p.root;
  const uint32_t* pi_s = nullptr;  // the round's folded codeword in shared memory, after round i0
  uint4* tree = p.next_tree;
  uint32_t* out_g = p.fold_out;
  for (int i = p.i0, it = 0; i >= 0; --i, ++it) {
    const uint32_t n = 1u << (p.log2_n0 + i), half = 1u << (i + p.lk);
    uint32_t* pairs = pi_s == pi_b ? pi_b : pi_a;
    uint32_t* next = pairs == pi_a ? pi_b : pi_a;
    if (warp == 0) {
      bb_challenge(wk, sh, root, p.rec + 72 * (size_t)it);
    } else {
      if (threadIdx.x >= 32 && threadIdx.x < 37) sums[(it + 1) & 1][threadIdx.x - 32] = 0;
      const uint32_t* tinv = p.tinv + (((size_t)1 << (p.log2_n0 + i)) - ((size_t)1 << p.log2_n0));
      for (uint32_t j = threadIdx.x - 32; j < n; j += kTreeThreads - 32) {
        E5 lo, hi;
        if (pi_s) {
          lo = ld_e5(pi_s, j);
          hi = ld_e5(pi_s, j + n);
        } else {
          lo = p.pi_base ? bb::e_from(p.pi[j]) : ld_e5(p.pi, j);
          hi = p.pi_base ? bb::e_from(p.pi[j + n]) : ld_e5(p.pi, j + n);
        }
        const E5 l = bb::e_scale(bb::e_add(lo, hi), bb::MONT_INV2);
        const E5 h = bb::e_scale(bb::e_sub(lo, hi), tinv[j]);
        st_e5(pairs, j, l);
        st_e5(pairs, j + n, bb::e_sub(h, l));
      }
    }
    __syncthreads();
    const E5 x = sh.t.x;
    // fold from the first thread up: row s of the next round's matrix is (out[s], out[s + n/2])
    const uint32_t rows = n > 1 ? n / 2 : 1;
    const int bits = p.log2_n0 + i - 1;
    for (uint32_t s = threadIdx.x; s < rows; s += kTreeThreads) {
      uint32_t w[10];
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const uint32_t j = s + q * rows;
        if (j >= n) break;
        const E5 f = bb::e_add(ld_e5(pairs, j), bb::e_mul(ld_e5(pairs, j + n), x));
        st_e5(out_g, j, f);
        st_e5(next, j, f);
#pragma unroll
        for (int e = 0; e < 5; ++e) w[5 * q + e] = bb::from_mont(f.c[e]);
      }
      if (i > 0) {  // n >= 2
        uint2* m = msg + 5 * (bits ? __brev(s) >> (32 - bits) : 0u);
#pragma unroll
        for (int e = 0; e < 5; ++e) m[e] = bi_from_lane(make_uint2(w[2 * e], w[2 * e + 1]));
      }
    }
    // fix and the next round's sum from the last thread down
    const uint32_t next_half = half >> 1;
    E5 part = bb::e_zero();
    for (uint32_t b = kTreeThreads - 1 - threadIdx.x; b < half; b += kTreeThreads) {
      const E5 lo = it ? ld_e5(poly, b) : ld_poly(b), hi = it ? ld_e5(poly, b + half) : ld_poly(b + half);
      const E5 v = bb::e_add(lo, bb::e_mul(x, bb::e_sub(hi, lo)));
      st_e5(poly, b, v);
      if (i > 0 && b < next_half) part = bb::e_add(part, bb::e_mul(ld_e5(p.heq, b), v));
    }
    if (i > 0) add_sums(part, sums[(it + 1) & 1]);
    __syncthreads();
    out_g += 5 * (size_t)n;
    pi_s = next;
    if (i > 0) {
      const uint32_t leaves = n / 2;
      // the claim and the next message by the last warp, which has no leaf to hash
      // unless there are eight of them
      auto next_message = [&] {
        if (warp != kTreeThreads / 32 - 1) return;
        bb_claim(sh);
        bb_message(sh, p.c, i - 1 + p.lk, (uint32_t)(sums[(it + 1) & 1][wk.lane % 5] % bb::P));
      };
      const bool busy = leaves == 8;
      if (!busy) next_message();
      hash_level_block<5>(wk, reinterpret_cast<const uint4*>(msg), 1, leaves, ts.a, tree, 1);
      __syncthreads();
      if (!busy) {
        root = tree_block(wk, ts.b, ts.a, ts.a, 1, tree + 2 * (size_t)leaves, leaves, 0, bits);
      } else {
        next_message();
        hash_level_block<8>(wk, ts.a, 1, leaves / 2, ts.b, tree + 2 * (size_t)leaves, 1);
        __syncthreads();
        root = tree_block(wk, ts.a, ts.b, ts.b, 1, tree + 3 * (size_t)leaves, leaves / 2, 0, bits - 1);
      }
      tree += 2 * (size_t)(2 * leaves);
    }
  }
  for (uint32_t q = threadIdx.x; q < (5u << p.lk); q += kTreeThreads) p.poly_out[q] = poly[q];
  tr_copy(p.t, &sh.t);
}

cudaError_t bb_launch_transcript_round(BbTranscript* t, const BbRoundConsts* c, int ri, const uint4* root_dev,
                                       unsigned long long* sums, int canonical, uint32_t* x_out, uint8_t* rec,
                                       bool first, bool early, cudaStream_t st) {
  const cudaError_t e =
      launch_chained(bb_transcript_round_kernel, 1, 32, 0, st, t, c, ri, root_dev, sums, canonical, x_out, rec, first, early);
  count_launch();
  return e;
}

cudaError_t bb_launch_tail(const BbTail& p, cudaStream_t st) {
  if (p.i0 < 0 || (1 << (p.log2_n0 + p.i0)) > kBbTailMax) return cudaErrorInvalidValue;
  const cudaError_t e = launch_chained(bb_tail_kernel, 1, kTreeThreads, 0, st, p);
  count_launch();
  return e;
}

}  // namespace bf
