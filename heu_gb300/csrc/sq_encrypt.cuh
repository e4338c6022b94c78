// Fixed-base encryption modulo n^2 in two digits (sqmod.cuh):
//   c = (1 + m n) h_s^r mod n^2   (encryptor.cc:26-56, evaluator.cc:25-28)
//
// A table entry Y = Y0 - Y1 n is kept as the integer Y0 and y = Y1 / Y0 mod n,
//   Y = Y0 (1 - y n) mod n^2,
// and the second factors multiply by adding their y: the chain of products
// runs over the integers Y0 alone (4 H^2 multiply-adds a product, half of a
// product modulo n^2), the y of the entries are summed, the plaintext's factor
// 1 + m n joins the sum, and one product at the end puts the sum in:
//   c = (P0 - P1 n)(1 - (sum y - m) n) = P0 - (P1 + P0 (sum y - m)) n.
// y is stored times rho, so the last product of digits is one reduction.
#pragma once
#include <cooperative_groups.h>

#include "paillier_ops.cuh"
#include "sqmod.cuh"

namespace hg {
inline namespace HG_SQ_SPACE {

// Shared words of a warp: two entries in flight and the sum of the y.
template <int TC, int L>
constexpr int kEncWords = 5 * SqLanes<TC, L>::kDigit;

__device__ __forceinline__ void cp_async(uint32_t* dst, const uint32_t* src, int bytes) {
  const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
  if (bytes == 16)
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(src) : "memory");
}

// The plaintext's magnitude in each chain's lanes; false where it is out of
// range (encryptor.cc:38-40: |m| <= n/2), and then 0.
template <int TC, int L>
__device__ __forceinline__ bool enc_plain(uint32_t (&A)[L], bool& neg, const KeyConst& kc, const EncArgs& a, size_t i,
                                          const SqLanes<TC, L>& g) {
  constexpr int H = TC * L;
  if (a.cd.kind == kCodecNone && a.m_mag == nullptr) {
    const int64_t v = a.m[i];
    const uint64_t u = abs_i64(v);
    neg = v < 0;
#pragma unroll
    for (int j = 0; j < L; ++j) {
      const int gi = g.t * L + j;
      A[j] = gi == 0 ? (uint32_t)u : gi == 1 ? (uint32_t)(u >> 32) : 0u;
    }
    return true;
  }
  bool bad = false;
  if (a.cd.kind != kCodecNone) {
    const EncodedPlain e = encode_plain(a.cd, a.m, i);
    neg = e.neg;
    bad = e.bad;
#pragma unroll
    for (int j = 0; j < L; ++j) A[j] = encoded_limb(e, g.t * L + j);
  } else {
    neg = a.m_neg[i] != 0;
    load_slice<L>(A, a.m_mag + i * H + g.t * L);
  }
  uint32_t half[L], d[L];
  load_slice<L>(half, kc.nhalf + g.t * L);
  const bool too_big = chain_sub<TC, L>(d, half, A) != 0u;
  if (too_big || bad) {
#pragma unroll
    for (int j = 0; j < L; ++j) A[j] = 0u;
  }
  return !(too_big || bad);
}

// One encryption per group of 2 TC lanes by kWarps warps of each block of a
// cluster of kBlocks: warp w multiplies the w-th share of the entries and warp 0
// combines the shares, so a short batch's chain of products is shorter.
// `area`: the warp's kEncWords, `carries` 32 words a warp.
template <int TC, int L, int kWarps, int kBlocks, class Mod>
__device__ __forceinline__ void sq_encrypt(const Mod& n, const KeyConst& kc, const EncArgs& a,
                                           uint32_t* __restrict__ out, size_t i, bool active, uint32_t* area,
                                           uint32_t* carries, uint32_t* err, const SqLanes<TC, L>& g) {
  constexpr int H = TC * L, S = 2 * H, kDigit = SqLanes<TC, L>::kDigit, V = SqLanes<TC, L>::kVec;
  const uint32_t np = kc.npn;
  constexpr int kShares = kWarps * kBlocks;
  const int slot = kWarps > 1 ? (int)(threadIdx.x >> 5) : 0;
  const int warp = kBlocks > 1 ? (int)(blockIdx.x % kBlocks) * kWarps + slot : slot;
  const size_t ent = (size_t)((1u << kc.w) - 1u);
  const uint32_t* ri = a.r + i * kc.rlimbs;
  // entry e: the table's for digit position e, one of the identity for a zero
  // digit, and past the positions the constant that a randomized ciphertext
  // (in the boundary's Montgomery form) still needs
  auto fetch = [&](int e, int buf) {
    const uint32_t* src;
    if (e >= kc.npos) {
      src = kc.rz;
    } else {
      const int off = e * kc.w;
      const uint32_t dg = get_bits(ri, kc.rlimbs, off, min(kc.w, kc.rbits - off));
      src = dg ? kc.table + ((size_t)e * ent + (dg - 1u)) * S : e == 0 ? kc.e0 : kc.e1;
    }
    src += g.c * H + g.t * L;
    uint32_t* dst = g.limb(area + buf * 2 * kDigit, g.c, 0);
#pragma unroll
    for (int v = 0; v < L / V; ++v) cp_async(dst + g.slice_at(v), src + v * V, V * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto arrived = [] {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
  };
  uint32_t* sum = g.limb(area + 4 * kDigit, 0, 0);  // of the y, chain 1's slices
  const int total = kc.npos + (a.mode == EncMode::kRandomize ? 1 : 0);
  int e = kShares > 1 ? total * warp / kShares : 0;
  const int end = kShares > 1 ? total * (warp + 1) / kShares : total;
  uint32_t x[L], carry = 0u;
  if (a.mode == EncMode::kRandomize && warp == 0) {
    const bool ok = raw_below<TC, L>(a.ct_in + i * S, kc.N);
    if (active && !ok && g.lane == g.base) atomicOr(err, kErrCtRange);
    if (e < end) fetch(e, 0);
    sq_from_raw<TC, L, S>(x, a.ct_in + i * S, n, np, g);
#pragma unroll
    for (int j = 0; j < L; ++j) {
      const int at = g.slice_at(j / V) + j % V;
      if (g.c == 1) sum[at] = 0u;
    }
  } else {
    // the first factor is an entry itself (the identity for an empty share)
    uint32_t s[L];
    const uint32_t* src = kc.e1;
    if (e < end) {
      const int off = e * kc.w;
      if (e >= kc.npos) {
        src = kc.rz;
      } else {
        const uint32_t dg = get_bits(ri, kc.rlimbs, off, min(kc.w, kc.rbits - off));
        src = dg ? kc.table + ((size_t)e * ent + (dg - 1u)) * S : e == 0 ? kc.e0 : kc.e1;
      }
    }
    if (e + 1 < end) fetch(e + 1, 0);
    ++e;
    load_slice<L>(s, src + g.c * H + g.t * L);
    if (g.c == 1) sq_put<TC, L>(sum, s, g);
#pragma unroll
    for (int j = 0; j < L; ++j) x[j] = g.c ? 0u : s[j];
  }
#pragma unroll 1
  for (int buf = 0; e < end; ++e, buf ^= 1) {
    arrived();
    if (e + 1 < end) fetch(e + 1, buf ^ 1);
    uint32_t* cur = area + buf * 2 * kDigit;
    if (g.c == 1) {
      uint32_t s[L], y[L];
      sq_get<TC, L>(s, sum, g);
      sq_get<TC, L>(y, g.limb(cur, 1, 0), g);
      s[0] = add_cc(s[0], y[0]);
#pragma unroll
      for (int j = 1; j < L; ++j) s[j] = addc_cc(s[j], y[j]);
      carry = addc(carry, 0u);
      sq_put<TC, L>(sum, s, g);
    }
    __syncwarp();
    sq_pass<TC, L, false>(x, x, g.limb(cur, 0, 0), 0u, 0u, x, nullptr, n, np, g);
  }
  if constexpr (kShares > 1) {
    // shares as a tree: warp w takes warp w + d's digits and sum, from another
    // block's shared memory where d reaches beyond its own
    namespace cg = cooperative_groups;
#pragma unroll 1
    for (int d = 1; d < kShares; d <<= 1) {
      if (warp % d == 0) {
        sq_stage<TC, L>(area, x, true, g);
        carries[slot * 32 + g.lane] = carry;
      }
      if (kBlocks > 1 && d >= kWarps)
        cg::this_cluster().sync();
      else
        __syncthreads();
      if (warp % (2 * d) == 0) {
        uint32_t* other = area + d * kEncWords<TC, L>;
        uint32_t* other_carries = carries + (slot + d) * 32;
        if constexpr (kBlocks > 1) {
          if (d >= kWarps) {
            const unsigned rank = (unsigned)((warp + d) / kWarps);
            other = cg::this_cluster().map_shared_rank(area, rank);
            other_carries = cg::this_cluster().map_shared_rank(carries + slot * 32, rank);
          }
        }
        if (g.c == 1) {
          uint32_t s[L], y[L];
          sq_get<TC, L>(s, sum, g);
          sq_get<TC, L>(y, g.limb(other + 4 * kDigit, 0, 0), g);
          s[0] = add_cc(s[0], y[0]);
#pragma unroll
          for (int j = 1; j < L; ++j) s[j] = addc_cc(s[j], y[j]);
          carry = addc(carry, other_carries[g.lane]);
          sq_put<TC, L>(sum, s, g);
        }
        uint32_t y0[L];
        sq_get<TC, L>(x, g.limb(other, g.c, 0), g);
        sq_get<TC, L>(y0, g.limb(other, 0, 0), g);
        sq_pass<TC, L, true>(x, x, g.limb(area, 0, 0), 0u, 0u, y0, g.limb(area, 1, 0), n, np, g);
      }
    }
    // the other blocks' shared memory has been read
    if constexpr (kBlocks > 1) cg::this_cluster().sync();
    if (warp != 0) return;
  }
  // sum - m rho, then X1 += X0 * sum
  uint32_t A[L], nn[L];
  bool neg = true;
#pragma unroll
  for (int j = 0; j < L; ++j) {
    A[j] = 0u;
    nn[j] = n[j];
  }
  if (a.mode == EncMode::kEncrypt) {
    const bool ok = enc_plain<TC, L>(A, neg, kc, a, i, g);
    if (active && !ok && g.lane == g.base) atomicOr(err, kErrPtRange);
  }
  __syncwarp();
  if (g.c == 1) sq_put<TC, L>(g.limb(area, 1, 0), A, g);
  load_slice<L>(A, (neg ? kc.rho2 : kc.nrho2) + g.t * L);
  uint32_t top = 0u;
#pragma unroll 1
  for (int k = 0; k < 2; ++k) {
    // k = 0: -m rho (-+rho^2 times |m|); k = 1: X0 times the whole sum
    __syncwarp();
    uint32_t z[L];
    sq_pass<TC, L, false, false>(z, A, g.limb(area, 1, 0), 0u, top, A, nullptr, n, np, g);
    if (k == 0) {
      uint32_t w[L];
      sq_get<TC, L>(w, sum, g);
      w[0] = add_cc(w[0], z[0]);
#pragma unroll
      for (int j = 1; j < L; ++j) w[j] = addc_cc(w[j], z[j]);
      carry = addc(carry, 0u);
      top = chain_settle<TC, L>(w, carry);
      if (g.c == 0) top = 0u;
      __syncwarp();
      if (g.c == 1) sq_put<TC, L>(g.limb(area, 1, 0), w, g);
#pragma unroll
      for (int j = 0; j < L; ++j) A[j] = __shfl_sync(kFull, x[j], g.c ? g.lane - TC : g.lane);
    } else {
      uint32_t w[L];
      chain_reduce_once<TC, L>(z, 0u, nn);
      const uint32_t over = chain_add<TC, L>(w, x, z);
      chain_reduce_once<TC, L>(w, over, nn);
      select_slice<L>(x, g.c == 1, w, x);
    }
  }
  uint32_t r[L];
  sq_to_raw<TC, L>(r, x, area, n, np, g);
  if (active) store_slice<L>(out + i * S + g.c * H + g.t * L, r);
}

}  // namespace HG_SQ_SPACE
}  // namespace hg
