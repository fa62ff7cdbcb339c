// Basefold::open with the Fiat–Shamir transcript on the device.
//
// The transcript (GenericChallenger over Keccak-256, p3/src/challenger.rs)
// and the round-polynomial scalars (eval.rs:89-111, eval_impr.rs:45-58,
// 116-127) live in an OpenState in device memory, so a whole open is one
// stream of kernels with no host round trip:
//  * open_observe_kernel observes the commitment root and the evaluation, as
//    the caller of open does (poly-commit/src/lib.rs:80-100);
//  * open_round_kernel is the transcript step of one large round; the fold,
//    fix and tree kernels of that round read the sampled challenge from the
//    state;
//  * open_tail_kernel runs every remaining round once the folded codeword has
//    at most a few thousand entries — fold + leaf hashes, Merkle levels, fix +
//    reduction and the transcript step, in one block separated by
//    __syncthreads — then observes the final polynomial (basefold.rs:196).
// The query positions (basefold.rs:200-203) are a serial chain of about 80
// Keccak digests, which the host computes far faster than one GPU thread, so
// they are sampled on the host from the returned transcript.
// The bytes produced are the same as the host-driven rounds'.
#include <cuda_runtime.h>

#include <cstdint>

#include "bf_internal.h"
#include "gf128.cuh"
#include "keccak.cuh"
#include "launch.cuh"

namespace bf {

namespace {

__device__ __forceinline__ uint4 one_dev() { return make_uint4(1u, 0u, 0u, 0xc2000000u); }

// The transcript is kept in shared memory and driven by one warp: the
// Keccak permutations run on all 32 lanes (WarpKeccak), the byte bookkeeping
// and the field arithmetic on lane 0, with __syncwarp between them.

// HashChallenger::flush: digest = keccak256(input); input = output = digest.
__device__ void warp_flush(const WarpKeccak& wk, DevTranscript& t) {
  __syncwarp();
  const int len = t.in_len;
  uint2 a = make_uint2(0, 0);
  for (int off = 0;; off += 136) {
    const int take = len - off < 136 ? len - off : 136;
    const bool last = take < 136;
    if (wk.lane < 17) {
      const int pos0 = 8 * wk.lane;
      uint2 w;
      if (pos0 + 8 <= take) {  // a whole message word (off and pos0 are multiples of 8)
        w = *reinterpret_cast<const uint2*>(t.in + off + pos0);
      } else {
        uint32_t h[2] = {0, 0};
        for (int b = 0; b < 8; ++b) {
          const int pos = pos0 + b;
          uint32_t v = pos < take ? t.in[off + pos] : 0u;
          if (last && pos == take) v ^= 0x01u;  // pad10*1 (original Keccak)
          h[b >> 2] |= v << (8 * (b & 3));
        }
        w = make_uint2(h[0], h[1]);
      }
      if (last && wk.lane == 16) w.y ^= 0x80000000u;  // last byte of the rate
      a = kx2(a, w);
    }
    a = wk.permute<false>(a);
    if (last) break;
  }
  __syncwarp();
  if (wk.lane < 4) {
    reinterpret_cast<uint2*>(t.out)[wk.lane] = a;
    reinterpret_cast<uint2*>(t.in)[wk.lane] = a;
  }
  if (wk.lane == 0) {
    t.out_len = 32;
    t.in_len = 32;
  }
  __syncwarp();
}

// CanObserve<u8> of the 16*N bytes of v (lane 0): append to the input, drop
// unread output.
template <int N>
__device__ void tr_observe(OpenState& o, const uint4 (&v)[N]) {
  DevTranscript& t = o.tr;
  t.out_len = 0;
  const int len = t.in_len;
  if (len + 16 * N > kTrMax) {
    o.status = 1;
    return;
  }
  if ((len & 15) == 0) {
#pragma unroll
    for (int k = 0; k < N; ++k) reinterpret_cast<uint4*>(t.in + len)[k] = v[k];
  } else {
#pragma unroll
    for (int k = 0; k < N; ++k) {
      const uint32_t w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
#pragma unroll
      for (int b = 0; b < 16; ++b) t.in[len + 16 * k + b] = (uint8_t)(w[b >> 2] >> (8 * (b & 3)));
    }
  }
  t.in_len = len + 16 * N;
}

// A field element from 16 sampled bytes, each popped from the end of the
// output, little-endian (challenger.rs sample, from_uniform_bytes.rs:20-26).
// Warp-collective; the element is returned on lane 0.
__device__ uint4 warp_sample_elem(const WarpKeccak& wk, OpenState& o) {
  __syncwarp();
  if (o.tr.out_len == 0) warp_flush(wk, o.tr);
  uint32_t w[4] = {0, 0, 0, 0};
  if (o.tr.out_len >= 16) {
    if (wk.lane == 0) {
      const int top = o.tr.out_len - 1;
#pragma unroll
      for (int k = 0; k < 16; ++k) w[k >> 2] |= (uint32_t)o.tr.out[top - k] << (8 * (k & 3));
      o.tr.out_len = top + 1 - 16;
    }
  } else {
    for (int k = 0; k < 16; ++k) {
      __syncwarp();
      if (o.tr.out_len == 0) warp_flush(wk, o.tr);
      if (wk.lane == 0) {
        const uint32_t byte = o.tr.out[--o.tr.out_len];
        w[k >> 2] |= byte << (8 * (k & 3));
      }
    }
  }
  __syncwarp();
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// The transcript step of round i in three parts, each warp-collective, so that only
// the middle one stands between a round's root and its challenge.
//
// EvalImprProver::compute_round_poly gives [c0, c1] (eval_impr.rs:116-127);
// EvalProver lifts it by delta = d * [1 - r, r - (1 - r)] = d * [1 + r, 1]
// in characteristic 2 (eval.rs:89-106), so the round polynomial is
// (c0 + c1 X)(d (1 + r) + d X): c0' = c0 d (1 + r), c2' = c1 d.  After the
// challenge x the EvalProver claim is c0 + c1 x and d becomes d (1 + r + x);
// the sumcheck claim (the round polynomial at x) is only read in the first
// round, so it is not carried.
//
// round_message: c0', c2' from S = sum_b half_eq[b] poly_lo[b] and the claim.
// Every lane computes the same scalars; the products are spread over the warp
// (gf_mul_warp2), two independent ones at a time.
__device__ void round_message(OpenState& o, bool first, uint4 r, uint4 r_inv, uint4 corr, uint4 S, uint4& rp0,
                              uint4& rp2) {
  const uint4 claim = first ? o.outer : o.inner;
  const uint4 delta = o.delta;
  const uint4 one_r = gf_add(one_dev(), r);
  uint4 c0, d0, t, c1;
  gf_mul_warp2(corr, S, delta, one_r, c0, d0);  // c0 = corr * S; d0 = delta (1 + r)
  gf_mul_warp2(one_r, c0, c0, d0, t, rp0);      // rp0 = c0 d0
  c1 = gf_add(gf_mul_warp(gf_add(claim, t), r_inv), c0);
  rp2 = gf_mul_warp(c1, delta);
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    o.c[0] = c0;
    o.c[1] = c1;
    o.c[2] = one_r;
  }
  __syncwarp();
}

// round_challenge: observes the root (a tree digest, interleaved) and the message,
// samples o.x; `rec` (global, 16-byte aligned) receives root, c0', c2'.
__device__ void round_challenge(const WarpKeccak& wk, OpenState& o, uint4 root_lo_bi, uint4 root_hi_bi, uint4 rp0,
                                uint4 rp2, uint4* rec) {
  if (wk.lane == 0) {
    Digest rt;
    rt.lo = root_lo_bi;
    rt.hi = root_hi_bi;
    rt = digest_bytes(rt);
    rec[0] = rt.lo;
    rec[1] = rt.hi;
    rec[2] = rp0;
    rec[3] = rp2;
    const uint4 m[4] = {rt.lo, rt.hi, rp0, rp2};
    tr_observe(o, m);  // root (basefold.rs:356), then [c0, c2] (sumcheck/src/lib.rs:97)
  }
  const uint4 x = warp_sample_elem(wk, o);
  if (wk.lane == 0) o.x = x;
  __syncwarp();
}

// round_claim: the claim and delta after the challenge.
__device__ void round_claim(OpenState& o) {
  const uint4 x = o.x, delta = o.delta, c0 = o.c[0], c1 = o.c[1], one_r = o.c[2];
  uint4 c1x, delta_next;
  gf_mul_warp2(c1, x, delta, gf_add(one_r, x), c1x, delta_next);
  __syncwarp();
  if ((threadIdx.x & 31) == 0) {
    o.inner = gf_add(c1x, c0);  // EvalProver::fix_last_var (eval.rs:108-111)
    o.delta = delta_next;
  }
  __syncwarp();
}

constexpr int kStateVecs = (int)(sizeof(OpenState) / sizeof(uint4));

__device__ __forceinline__ void state_load(OpenState& sh, const OpenState* g) {
  const uint4* src = reinterpret_cast<const uint4*>(g);
  uint4* dst = reinterpret_cast<uint4*>(&sh);
  for (int k = threadIdx.x; k < kStateVecs; k += blockDim.x) dst[k] = __ldcg(src + k);
}
__device__ __forceinline__ void state_store(OpenState* g, const OpenState& sh) {
  const uint4* src = reinterpret_cast<const uint4*>(&sh);
  uint4* dst = reinterpret_cast<uint4*>(g);
  for (int k = threadIdx.x; k < kStateVecs; k += blockDim.x) dst[k] = src[k];
}

}  // namespace

__global__ void __launch_bounds__(32) open_observe_kernel(OpenState* S, const uint4* root, const uint4* value) {
  __shared__ OpenState sh;
  state_load(sh, S);
  __syncthreads();
  if (threadIdx.x == 0) {
    if (root) {  // a tree root, stored interleaved
      const Digest rb = digest_bytes(load_digest(root, 0));
      const uint4 m[2] = {rb.lo, rb.hi};
      tr_observe(sh, m);
    }
    if (value) {
      const uint4 m[1] = {value[0]};
      tr_observe(sh, m);
      sh.outer = m[0];
    }
  }
  __syncthreads();
  state_store(S, sh);
}

// From the second round on, the launch before this one is a tree's, and a block of
// this grid starts only after every block of that one has waited for all launches
// before it: the state and the reduction S, which those wrote, are read (past L1)
// and the message made before the wait, which is left for the root alone (an early
// reader, under the rules of launch.cuh).  From the
// tree's end to this kernel's end measured 3.9 us on GB300, 7.2 with everything after
// the wait.
__global__ void __launch_bounds__(32) open_round_kernel(OpenState* S, int i, int d, const uint4* scal,
                                                        const uint4* root, const uint4* Sred, uint8_t* rec) {
  __shared__ OpenState sh;
  const WarpKeccak wk;
  const bool first = i == d - 1;
  if (first) chain_wait();
  state_load(sh, S);
  __syncwarp();
  if (!first) round_claim(sh);
  uint4 rp0, rp2;
  round_message(sh, first, __ldcg(scal + 3 * i), __ldcg(scal + 3 * i + 1), __ldcg(scal + 3 * i + 2), __ldcg(Sred), rp0,
                rp2);
  if (!first) chain_wait();
  round_challenge(wk, sh, root[0], root[1], rp0, rp2, reinterpret_cast<uint4*>(rec));
  state_store(S, sh);
}

// The last rounds in one block of eight warps.  Rounds whose fold has at most
// kTailShared outputs keep the folded codeword, the leaf messages and the tree
// levels in shared memory (a level read back from global memory costs an L2
// round trip), hash each level in the form that is fastest for its count
// (hash_level_block), and multiply by the twiddles, which need no challenge,
// on warps 1..7 while warp 0 samples the challenge: after it a fold output is one
// product, and the next reduction is a + x b of two sums that are ready.  The claim
// and the next round's message are made while the leaves are hashed, by a warp
// that has no hash there.  Bound by the chain of dependent permutations
// (one per level, leaf and transcript step).  Measured on GB300 for the last nine
// rounds of an open (fold outputs from 2^9): 172 us, 191 with the message and the
// claim between root and challenge and a second product in the next reduction;
// with one thread per leaf and the codeword and levels in global memory, 262 for
// the last eight.
constexpr int kTailShared = 512, kTailPoly = 128;

__global__ void __launch_bounds__(kTailThreads, 1) open_tail_kernel(TailParams P) {
  static_assert(kTailThreads == kTreeThreads, "the tail hashes levels with hash_level_block");
  __shared__ OpenState sh;
  __shared__ uint4 pi_a[2 * kTailShared], pi_b[kTailShared];  // (lo', hi' - lo') pairs of a fold's input
  __shared__ uint4 msg[kTailShared];                          // a fold's outputs as interleaved lanes
  __shared__ TreeShared ts;
  __shared__ uint4 poly_s[kTailPoly];            // the polynomial once it fits
  __shared__ __align__(16) uint32_t sums[2][4];  // the next reduction is sums[0] + x sums[1]
  __shared__ uint4 rp[2];                        // the round's message
  const int d = P.d;
  const size_t c = (size_t)1 << P.log2_c;
  const WarpKeccak wk;
  const int warp = threadIdx.x >> 5;
  const bool early = P.i0 >= 0 && P.i0 < d - 1;  // after launched rounds: see open_round_kernel
  if (!early) chain_wait();
  state_load(sh, P.state);
  if (threadIdx.x < 8) sums[threadIdx.x >> 2][threadIdx.x & 3] = 0;
  __syncthreads();
  auto message = [&](int i, uint4 S) {  // one warp
    uint4 rp0, rp2;
    round_message(sh, i == d - 1, __ldcg(P.scal + 3 * i), __ldcg(P.scal + 3 * i + 1), __ldcg(P.scal + 3 * i + 2), S, rp0,
                  rp2);
    if (wk.lane == 0) {
      rp[0] = rp0;
      rp[1] = rp2;
    }
  };
  if (warp == 0 && P.i0 >= 0) {
    if (early) round_claim(sh);
    message(P.i0, __ldcg(P.S_i0));
  }
  if (early) chain_wait();
  const uint4* root = P.root_i0;  // the round's tree root
  const uint4* pi_s = nullptr;    // the round's folded codeword in shared memory, if it is there
  const uint4* poly = P.i0 == d - 1 ? P.poly_first : P.poly;
  __syncthreads();
  int k = 0;
  for (int i = P.i0; i >= 0; --i, ++k) {
    const size_t ni = c << i;
    const bool small = ni <= (size_t)kTailShared;
    const uint4* pi_in = (i == d - 1) ? P.pi_first : P.pi_fold + c * (((size_t)1 << d) - ((size_t)1 << (i + 2)));
    uint4* pi_out = P.pi_fold + c * (((size_t)1 << d) - ((size_t)1 << (i + 1)));
    const uint4* tlo = P.tw->lo[d - 1 - i];
    const uint4* thi = P.tw->hi[d - 1 - i];
    uint4* pairs = pi_s == pi_b ? pi_b : pi_a;
    uint4* next = pairs == pi_a ? pi_b : pi_a;
    const uint32_t half = 1u << i, next_half = half >> 1;
    // ---- the challenge (warp 0); meanwhile the other warps interpolate and add up
    //      sum heq lo and sum heq (hi + lo) over the next round's range ----
    if (warp == 0) {
      round_challenge(wk, sh, root[0], root[1], rp[0], rp[1], reinterpret_cast<uint4*>(P.result + 64 * (size_t)k));
    } else {
      if (small) {
        const uint4* src = pi_s ? pi_s : pi_in;
        for (uint32_t t = threadIdx.x - 32; t < ni; t += blockDim.x - 32) {
          const uint4 tw = gf_add(tlo[t & 4095], thi[t >> 12]);
          const uint4 lo = src[2 * t], hi = gf_add(src[2 * t + 1], lo);
          const uint4 l = gf_add(lo, gf_mul(hi, tw));
          pairs[2 * t] = l;
          pairs[2 * t + 1] = gf_add(hi, l);
        }
      }
      uint4 part[2] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
      for (uint32_t e = blockDim.x - 1 - threadIdx.x; e < 2 * next_half; e += blockDim.x - 32) {
        const uint32_t q = e & 1u, b = e >> 1;
        const uint4 lo = poly[b];
        part[0] = gf_add(part[0], gf_mul(P.heq[b], q ? gf_add(poly[b + half], lo) : lo));
      }
      // a thread's items all have the parity of its first (the stride is even)
      if ((threadIdx.x & 1u) == 0) {
        part[1] = part[0];
        part[0] = make_uint4(0, 0, 0, 0);
      }
      if (next_half) {
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          part[q] = warp_xor(part[q]);
          if (wk.lane == 0) atomic_xor4(sums[q], part[q]);
        }
      }
    }
    __syncthreads();
    const uint4 x = sh.x;
    uint4* leaves = nullptr;
    if (i > 0)
      leaves = P.pi_trees + 2 * ((c << 1) * (((size_t)1 << (d - 1)) - ((size_t)1 << i)) - (size_t)(d - 1 - i));
    // ---- fold from the first thread up, fix (+ next reduction) from the last down ----
    if (small) {
      for (uint32_t t = threadIdx.x; t < ni; t += blockDim.x) {
        const uint4 f = gf_add(pairs[2 * t], gf_mul(pairs[2 * t + 1], x));
        pi_out[t] = f;
        next[t] = f;
        const uint2 m0 = bi_from_lane(make_uint2(f.x, f.y)), m1 = bi_from_lane(make_uint2(f.z, f.w));
        msg[t] = make_uint4(m0.x, m0.y, m1.x, m1.y);
      }
      pi_s = next;
    } else {
      for (size_t t = threadIdx.x; t < ni; t += blockDim.x) {
        const uint4 tw = gf_add(tlo[t & 4095], thi[t >> 12]);
        uint4 lo = pi_in[2 * t], hi = pi_in[2 * t + 1];
        hi = gf_add(hi, lo);
        lo = gf_add(lo, gf_mul(hi, tw));
        pi_out[t] = gf_add(lo, gf_mul(gf_add(hi, lo), x));
      }
    }
    uint4* fixed = half <= (uint32_t)kTailPoly ? poly_s : P.poly;
    for (uint32_t b = blockDim.x - 1 - threadIdx.x; b < half; b += blockDim.x) {
      const uint4 lo = poly[b], hi = poly[b + half];
      fixed[b] = gf_add(lo, gf_mul(x, gf_add(hi, lo)));
    }
    poly = fixed;
    __syncthreads();
    // ---- the next round's leaves and Merkle tree ----
    if (i > 0) {
      size_t n = ni / 2;
      auto next_message = [&] {  // by the last warp, which hashes nothing unless 8 or 256 hashes are due
        if (warp != kTailThreads / 32 - 1) return;
        round_claim(sh);
        uint4* a = reinterpret_cast<uint4*>(sums);
        const uint4 S = gf_add(a[0], gf_mul_warp(a[1], x));
        __syncwarp();
        if (wk.lane < 2) a[wk.lane] = make_uint4(0, 0, 0, 0);
        message(i - 1, S);
      };
      if (small) {
        int levels = P.log2_c + i - 1;
        const bool busy = n == 8 || n == 256;
        if (!busy) next_message();
        hash_level_block<4>(wk, msg, 1, (uint32_t)n, ts.a, leaves, 1);
        __syncthreads();
        if (!busy) {
          root = tree_block(wk, ts.b, ts.a, ts.a, 1, leaves + 2 * n, n, 0, levels);
        } else {
          next_message();
          hash_level_block<8>(wk, ts.a, 1, (uint32_t)n / 2, ts.b, leaves + 2 * n, 1);
          __syncthreads();
          root = tree_block(wk, ts.a, ts.b, ts.b, 1, leaves + 3 * n, n / 2, 0, levels - 1);
        }
      } else {
        next_message();
        for (size_t s = threadIdx.x; s < n; s += blockDim.x)
          store_digest(leaves, s, hash_pair(pi_out[2 * s], pi_out[2 * s + 1]));
        __syncthreads();
        uint4* cur = leaves;
        int kn = P.log2_c + i - 1;
        for (; kn > kTreeBlockLog; --kn, n >>= 1) {
          const size_t h = n >> 1;
          uint4* nxt = cur + 2 * n;
          for (size_t s = threadIdx.x; s < h; s += blockDim.x)
            store_digest(nxt, s, hash_node(load_digest(cur, s), load_digest(cur, s + h)));
          __syncthreads();
          cur = nxt;
        }
        root = tree_block(wk, ts.a, ts.b, cur, 1, cur + 2 * n, n, 0, kn);
      }
    }
  }
  // ---- final polynomial (basefold.rs:196) ----
  if (threadIdx.x == 0) {
    const uint4 fin = poly[0];
    reinterpret_cast<uint4*>(P.result + 64 * (size_t)k)[0] = fin;
    const uint4 m[1] = {fin};
    tr_observe(sh, m);
    // the reference's debug self-check encode0(final_poly) == pi (basefold.rs:198):
    // every entry of the last folded codeword is the final polynomial
    if (P.i0 >= 0) {
      const uint4* pi0 = P.pi_fold + c * (((size_t)1 << d) - 2);
      for (size_t t = 0; t < c; ++t) {
        const uint4 e = pi0[t];
        if (e.x != fin.x || e.y != fin.y || e.z != fin.z || e.w != fin.w) sh.status |= 2;
      }
    }
  }
  __syncthreads();
  state_store(P.state, sh);
}

namespace {

// One round of the product sumcheck's transcript by one warp (see
// launch_sumcheck_round): the sums c0, c2, c3 are the same in every lane.
__device__ __forceinline__ void sumcheck_step(const WarpKeccak& wk, OpenState& sh, int k, uint4 c0, uint4 c2, uint4 c3,
                                              uint8_t* rec) {
  // k = 2: compressed [c0, c2] (the pair scalar is ONE, quadratic.rs:118); k = 3:
  // [c0, c2, c3]
  if (wk.lane == 0) {
    uint4* r = reinterpret_cast<uint4*>(rec);
    r[0] = c0;
    r[1] = c2;
    if (k == 3) {
      r[2] = c3;
      const uint4 m[3] = {c0, c2, c3};
      tr_observe(sh, m);
    } else {
      const uint4 m[2] = {c0, c2};
      tr_observe(sh, m);
    }
  }
  const uint4 x = warp_sample_elem(wk, sh);  // valid on lane 0
  if (wk.lane == 0) {
    reinterpret_cast<uint4*>(rec)[k] = x;
    sh.x = x;
    sh.c[0] = c0;
    sh.c[1] = c2;
    sh.c[2] = c3;
  }
  __syncwarp();
}

// The claim after the challenge: horner over the round polynomial at x.  The message
// does not need it, so this is left to the next step (one warp).
__device__ __forceinline__ void sumcheck_claim(OpenState& sh, int k) {
  // k = 2: round polynomial [c0, sc - 2 c0 - c2 = sc + c2, c2]; k = 3: [c0, sc + c2 +
  // c3, c2, c3]
  const uint4 sc = sh.outer, x = sh.x, c0 = sh.c[0], c2 = sh.c[1], c3 = sh.c[2];
  const uint4 c1 = (k == 3) ? gf_add(sc, gf_add(c2, c3)) : gf_add(sc, c2);
  uint4 acc_h = (k == 3) ? c3 : c2;
  if (k == 3) acc_h = gf_add(gf_mul_warp(acc_h, x), c2);
  acc_h = gf_add(gf_mul_warp(acc_h, x), c1);
  acc_h = gf_add(gf_mul_warp(acc_h, x), c0);
  __syncwarp();
  if ((threadIdx.x & 31) == 0) sh.outer = acc_h;
  __syncwarp();
}

}  // namespace

// Product sumcheck round (warp): c = [c0, c2, c3] from the device sums, which
// it clears for the fix that accumulates the next round's.
// After the first round the launch before this one is a fix's, whose blocks wait for
// the round's before it: the state is read, and its claim brought up to date, before
// the wait (see open_round_kernel).
__global__ void __launch_bounds__(32) sumcheck_round_kernel(OpenState* S, int k, bool first, uint32_t* acc,
                                                            uint8_t* rec) {
  __shared__ OpenState sh;
  const WarpKeccak wk;
  if (first) chain_wait();
  state_load(sh, S);
  __syncwarp();
  if (!first) {
    sumcheck_claim(sh, k);
    chain_wait();
  }
  uint4* a = reinterpret_cast<uint4*>(acc);
  const uint4 c0 = a[0], c2 = a[1], c3 = a[2];
  __syncwarp();
  if (wk.lane < 3) a[wk.lane] = make_uint4(0, 0, 0, 0);
  sumcheck_step(wk, sh, k, c0, c2, c3, rec);
  __syncthreads();
  state_store(S, sh);
}

// The last m rounds (at most kSumcheckTailLog) in one block (an early reader as
// above): transcript step,
// fix and the next round's sums, with the polynomials in shared memory.  The
// products of a round are spread over the threads one by one (an output of the
// fix, then the factors and the terms of a pair's sums), since a thread that
// takes a whole pair runs up to 13 products of 0.65 us one after another.
// Measured on GB300: a sumcheck over 2^14 points, K = 2 159 us (216 with two
// launches per round throughout), K = 3 222 us (312).
template <int K>
__global__ void __launch_bounds__(kTailThreads, 1) sumcheck_tail_kernel(SumcheckTail p) {
  constexpr int kMax = 1 << (kSumcheckTailLog - 1);  // outputs of the first fix
  __shared__ OpenState sh;
  __shared__ uint4 f[K][kMax];                          // the fixed polynomials
  __shared__ uint4 quad[K == 3 ? 3 * (kMax / 2) : 1];  // K = 3: b1 b2, lo1 lo2, cross of every pair
  __shared__ __align__(16) uint32_t sums[2][12];       // this round's c0, c2, c3 and the next one's
  const WarpKeccak wk;
  const uint32_t tid = threadIdx.x;
  if (p.first) chain_wait();
  state_load(sh, p.state);
  __syncthreads();
  if (!p.first) {
    if (tid < 32) sumcheck_claim(sh, K);
    chain_wait();
  }
  if (tid < 12) sums[0][tid] = p.acc[tid];
  __syncthreads();
  // item i of a round's terms adds v to coefficient q; a warp whose items all
  // have one q reduces first
  auto add_term = [&](uint4 v, int q, bool whole_warp, uint32_t* acc) {
    if (whole_warp) {
      v = warp_xor(v);
      if (wk.lane == 0) atomic_xor4(acc + 4 * q, v);
    } else {
      atomic_xor4(acc + 4 * q, v);
    }
  };
  for (int round = p.m - 1; round >= 0; --round) {
    const int it = p.m - 1 - round;
    const uint32_t half = 1u << round, nh = half >> 1;
    uint32_t* next = sums[(it + 1) & 1];
    if (tid < 32) {
      const uint4* c = reinterpret_cast<const uint4*>(sums[it & 1]);
      sumcheck_step(wk, sh, K, c[0], c[1], c[2], p.rec + 16 * (size_t)(K + 1) * it);
    } else if (tid < 44) {
      next[tid - 32] = 0;
    }
    __syncthreads();
    const uint4 x = sh.x;
    if (tid >= kTailThreads - 32) sumcheck_claim(sh, K);  // the warp with the fewest outputs
    // fix: output b of polynomial j
    uint4 out[(K * kMax + kTailThreads - 1) / kTailThreads];
#pragma unroll
    for (int q = 0; q < (K * kMax + kTailThreads - 1) / kTailThreads; ++q) {
      const uint32_t e = tid + q * kTailThreads;
      if (e >= K * half) break;
      const uint32_t j = e >> round, b = e & (half - 1);
      const uint4 lo = it ? f[j][b] : p.in[j][b], hi = it ? f[j][b + half] : p.in[j][b + half];
      out[q] = gf_add(lo, gf_mul(x, gf_add(hi, lo)));
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < (K * kMax + kTailThreads - 1) / kTailThreads; ++q) {
      const uint32_t e = tid + q * kTailThreads;
      if (e < K * half) f[e >> round][e & (half - 1)] = out[q];
    }
    __syncthreads();
    if (round == 0) break;
    const bool whole = nh >= 32;
    if (K == 3) {  // the pairs' factors: b1 b2, lo1 lo2 and hi1 hi2
      for (uint32_t e = tid; e < 3 * nh; e += kTailThreads) {
        const uint32_t t = e >> (round - 1), b = e & (nh - 1);
        const uint4 l1 = f[1][b], h1 = f[1][b + nh], l2 = f[K - 1][b], h2 = f[K - 1][b + nh];
        const uint4 u = t == 0 ? gf_add(l1, h1) : t == 1 ? l1 : h1, v = t == 0 ? gf_add(l2, h2) : t == 1 ? l2 : h2;
        quad[t * (kMax / 2) + b] = gf_mul(u, v);
      }
      __syncthreads();
      for (uint32_t e = tid; e < 4 * nh; e += kTailThreads) {
        const uint32_t t = e >> (round - 1), b = e & (nh - 1);
        const uint4 b12 = quad[b], lo12 = quad[kMax / 2 + b], hi12 = quad[kMax + b];
        const uint4 l0 = f[0][b], b0 = gf_add(l0, f[0][b + nh]);
        // c0 = lo0 lo12; c2 = b0 cross + lo0 b12, cross = hi12 + lo12 + b12; c3 = b0 b12
        const uint4 u = (t == 0 || t == 2) ? l0 : b0;
        const uint4 v = t == 0 ? lo12 : t == 1 ? gf_add(gf_add(hi12, lo12), b12) : b12;
        add_term(gf_mul(u, v), t == 0 ? 0 : t == 3 ? 2 : 1, whole, next);
      }
    } else {
      for (uint32_t e = tid; e < 2 * nh; e += kTailThreads) {
        const uint32_t t = e >> (round - 1), b = e & (nh - 1);
        const uint4 l0 = f[0][b], l1 = f[1][b];
        const uint4 u = t ? gf_add(l0, f[0][b + nh]) : l0, v = t ? gf_add(l1, f[1][b + nh]) : l1;
        add_term(gf_mul(u, v), (int)t, whole, next);
      }
    }
    __syncthreads();
  }
  if (tid < K) reinterpret_cast<uint4*>(p.rec + 16 * (size_t)(K + 1) * p.m)[tid] = f[tid][0];
  state_store(p.state, sh);
}

cudaError_t launch_sumcheck_tail(const SumcheckTail& p, int k, cudaStream_t st) {
  if ((k != 2 && k != 3) || p.m < 1 || p.m > kSumcheckTailLog) return cudaErrorInvalidValue;
  const cudaError_t e =
      launch_chained(k == 2 ? sumcheck_tail_kernel<2> : sumcheck_tail_kernel<3>, 1, kTailThreads, 0, st, p);
  count_launch();
  return e;
}

cudaError_t launch_sumcheck_round(OpenState* s, int k, bool first, uint32_t* acc, uint8_t* rec, cudaStream_t st) {
  if (k != 2 && k != 3) return cudaErrorInvalidValue;
  const cudaError_t e = launch_chained(sumcheck_round_kernel, 1, 32, 0, st, s, k, first, acc, rec);
  count_launch();
  return e;
}

cudaError_t launch_open_observe(OpenState* s, const uint4* root, const uint4* value, cudaStream_t st) {
  open_observe_kernel<<<1, 32, 0, st>>>(s, root, value);
  count_launch();
  return cudaGetLastError();
}

cudaError_t launch_open_round(OpenState* s, int i, int d, const uint4* scal, const uint4* root, const uint4* S,
                              uint8_t* rec, cudaStream_t st) {
  const cudaError_t e = launch_chained(open_round_kernel, 1, 32, 0, st, s, i, d, scal, root, S, rec);
  count_launch();
  return e;
}

cudaError_t launch_open_tail(const TailParams& p, cudaStream_t st) {
  const cudaError_t e = launch_chained(open_tail_kernel, 1, kTailThreads, 0, st, p);
  count_launch();
  return e;
}

}  // namespace bf
