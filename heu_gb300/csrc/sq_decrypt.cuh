// CRT decryption's pieces besides the exponentiation kernel of
// decrypt_kernels.cu: the tail that both it and the batch kernel end with, and
// the batch kernel's exponentiation.
#pragma once
#include "paillier_ops.cuh"
#include "sqmod.cuh"

namespace hg {
inline namespace HG_SQ_SPACE {

// m_p = z_p c1_p + c2_p mod p, the same for q, then the CRT combination
//   h = (m_q - m_p) p^-1 mod q, m = m_p + p h
// and the sign fold m > n/2 => m - n (decryptor.cc:49-52).  8 lanes per
// ciphertext, `z` its 2 H digits, `mm` 2 H words of shared memory.
template <int LT>
__device__ __forceinline__ void dec_tail(const KeyConst& kc, const SecConst& sc, const uint32_t* z, size_t i,
                                         bool active, uint32_t* mm, int64_t* __restrict__ out_i64,
                                         uint8_t* __restrict__ out_ovf, uint32_t* __restrict__ out_mag,
                                         uint8_t* __restrict__ out_neg, const Codec& cd) {
  constexpr int TP = 8, H = TP * LT, W = 2 * LT;
  const Group<TP> g;
  uint32_t P[LT], Q[LT], a[LT], b[LT], mp[LT], mq[LT];
  load_slice<LT>(P, sc.P[0] + g.t * LT);
  load_slice<LT>(Q, sc.P[1] + g.t * LT);
  load_slice<LT>(a, z + g.t * LT);
  load_slice<LT>(b, sc.c1[0] + g.t * LT);
  mont_mul<TP, LT>(mp, a, b, P, sc.np1[0], g);
  load_slice<LT>(b, sc.c2[0] + g.t * LT);
  mod_add<TP, LT>(mp, mp, b, P, g);
  load_slice<LT>(a, z + H + g.t * LT);
  load_slice<LT>(b, sc.c1[1] + g.t * LT);
  mont_mul<TP, LT>(mq, a, b, Q, sc.np1[1], g);
  load_slice<LT>(b, sc.c2[1] + g.t * LT);
  mod_add<TP, LT>(mq, mq, b, Q, g);
  // m_p mod q (p < 2q), then h
  reduce_once<TP, LT>(a, mp, 0u, Q, g);
  mod_sub<TP, LT>(mq, mq, a, Q, g);
  load_slice<LT>(b, sc.pinvqR + g.t * LT);
  mont_mul<TP, LT>(mq, mq, b, Q, sc.np1[1], g);
  // m = m_p + p h: rows of p, the lowest limb leaves in every step
  {
    uint32_t E[LT], O[LT], T[LT], ov = 0u, c1 = 0u;
#pragma unroll
    for (int j = 0; j < LT; ++j) {
      E[j] = mp[j];
      O[j] = 0u;
    }
#pragma unroll 1
    for (int owner = 0; owner < TP; ++owner) {
#pragma unroll
      for (int j = 0; j < LT; j += 2) {
        row_mac<LT>(E, O, ov, c1, P, __shfl_sync(kFull, mq[j], owner, TP));
        if (g.t == 0) mm[owner * LT + j] = E[0];
        shift_limb<TP, LT>(E, ov, c1, g);
        row_mac<LT>(O, E, ov, c1, P, __shfl_sync(kFull, mq[j + 1], owner, TP));
        if (g.t == 0) mm[owner * LT + j + 1] = O[0];
        shift_limb<TP, LT>(O, ov, c1, g);
      }
    }
    (void)settle<TP, LT>(T, E, O, ov, c1, g);
    store_slice<LT>(mm + H + g.t * LT, T);
  }
  __syncwarp();
  uint32_t M[W], X[W], D[W];
  load_slice<W>(M, mm + g.t * W);
  load_slice<W>(X, kc.nhalf + g.t * W);
  const bool gt = sub_full<TP, W>(D, X, M, g) != 0u;
  load_slice<W>(X, kc.n + g.t * W);
  (void)sub_full<TP, W>(D, X, M, g);
  select_slice<W>(M, gt, D, M);
  __syncwarp();
  store_slice<W>(mm + g.t * W, M);
  __syncwarp();
  if (cd.kind != kCodecNone) {
    if (active && g.t == 0) decode_plain<2 * H>(cd, mm, gt, i, out_i64, out_ovf);
    return;
  }
  if (out_mag) {
    if (active) store_slice<W>(out_mag + i * (2 * H) + g.t * W, M);
    if (active && g.t == 0) out_neg[i] = gt ? 1 : 0;
  }
  if (out_i64) {
    uint32_t high = 0u;
#pragma unroll
    for (int j = 0; j < W; ++j)
      if (g.t != 0 || j >= 2) high |= M[j];
    const uint32_t B = __ballot_sync(kFull, high != 0u);
    bool fits = ((B >> g.base) & 0xffu) == 0u;
    if (active && g.t == 0) {
      const uint64_t mag = (uint64_t)M[0] | ((uint64_t)M[1] << 32);
      fits = fits && (gt ? mag <= (1ull << 63) : mag < (1ull << 63));
      out_i64[i] = (int64_t)(gt ? (uint64_t)0 - mag : mag);
      if (out_ovf) out_ovf[i] = fits ? 0 : 1;
    }
  }
}

// Digits of the power -> its digit 1 in chain 1: digit 0 is 1, or a multiple
// of p where p divides c: such a c decrypts as it always did, through the
// value that stands for it.
template <int TC, int L>
__device__ __forceinline__ void dec_check(uint32_t (&x)[L], const SecConst& sc, int side, const SqLanes<TC, L>& g) {
  uint32_t any = x[0] ^ (g.t == 0 ? 1u : 0u);
#pragma unroll
  for (int j = 1; j < L; ++j) any |= x[j];
  const uint32_t mask = (1u << TC) - 1u;
  const bool zero = ((__ballot_sync(kFull, any != 0u) >> g.base) & mask) != 0u;
  if (zero) load_slice<L>(x, sc.vz[side] + g.t * L);
}

// x in Montgomery form -> digit 1 of the power in chain 1.
template <int TC, int L, class Mod>
__device__ __forceinline__ void dec_digit(uint32_t (&x)[L], const SecConst& sc, int side, const Mod& n, uint32_t np,
                                          const SqLanes<TC, L>& g) {
  sq_redc<TC, L>(x, x, n, np, g);
  dec_check<TC, L>(x, sc, side, g);
}

// The exponentiation in the batch kernel: the two sides of a ciphertext sit in
// neighbouring groups of one warp, so every group must square and multiply in
// the same steps: windows of kBatchDecWindow bits at fixed places (sc.fprog),
// all powers 0 .. 2^w - 1 in the table; 5% more work than sliding windows.
// Writes digit 1 of this group's side to zs (H words).

template <int TC, int L>
__device__ __forceinline__ void dec_pow_fixed(const KeyConst& kc, const SecConst& sc, int side,
                                              const uint32_t* __restrict__ ct, size_t i, bool active, uint32_t* tb,
                                              uint32_t* area, uint32_t* zs, uint32_t* err,
                                              const SqLanes<TC, L>& g) {
  constexpr int H = TC * L, kTab = 1 << kBatchDecWindow;
  const uint32_t np = sc.np1[side];
  const uint8_t* prog = sc.fprog[side];
  const uint32_t* src = ct + i * (4 * H);
  const bool ok = raw_below<TC, 2 * L>(src, kc.N);
  if (active && !ok && side == 0 && g.lane == g.base) atomicOr(err, kErrCtRange);
  uint32_t n[L], x[L];
  load_slice<L>(n, sc.P[side] + g.t * L);
  load_slice<L>(x, sc.one[side] + g.c * H + g.t * L);
  table_store<L>(tb, 0, g.lane, x);
  sq_from_raw<TC, L, 4 * H>(x, src, n, np, g);
  table_store<L>(tb, 1, g.lane, x);
  // step s < kTab - 2 makes power s + 2; then w squarings and a product a window
  const int steps = kTab - 2 + (sc.fwin - 1) * (kBatchDecWindow + 1);
#pragma unroll 1
  for (int s = 0; s < steps; ++s) {
    int e = -1;  // -1: square, else multiply by slot e
    if (s < kTab - 2) {
      if (s & 1)
        e = 1;
      else
        table_load<L>(x, tb, (s + 2) >> 1, g.lane);
    } else {
      const int q = s - (kTab - 2), win = q / (kBatchDecWindow + 1);
      if (q == 0) table_load<L>(x, tb, prog[0], g.lane);
      if (q - win * (kBatchDecWindow + 1) == kBatchDecWindow) e = prog[win + 1];
    }
    sq_stage<TC, L>(area, x, __any_sync(kFull, e >= 0), g);
    if (!__any_sync(kFull, e >= 0)) {
      sq_pass<TC, L, false>(x, x, g.limb(area, 0, 0), (uint32_t)g.c, 0u, x, nullptr, n, np, g);
    } else {
      uint32_t y0[L];
      table_load<L>(x, tb, e, g.lane);
      table_load<L>(y0, tb, e, g.lane - g.c * TC);
      sq_pass<TC, L, true>(x, x, g.limb(area, 0, 0), 0u, 0u, y0, g.limb(area, 1, 0), n, np, g);
    }
    if (s < kTab - 2) table_store<L>(tb, s + 2, g.lane, x);
  }
  dec_digit<TC, L>(x, sc, side, n, np, g);
  if (g.c == 1) {
#pragma unroll
    for (int j = 0; j < L; ++j) zs[g.t * L + j] = x[j];
  }
}

}  // namespace HG_SQ_SPACE
}  // namespace hg
