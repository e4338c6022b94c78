// Arithmetic modulo the square of an odd number n of H limbs, for sm_103a.
//
// A residue is held as two digits to the base n, X = X0 - X1 n mod n^2 with
// 0 <= X0, X1 < 2^(32 H) (not necessarily below n).  With rho = 2^(32 (H+1))
// one Montgomery reduction modulo n gives both the next digit 0 and what it
// owes to digit 1:
//   X0 Y0 + m n = Z0 rho,  0 <= m < rho
//   X Y / rho = Z0 - Z1 n,  Z1 = (X0 Y1 + X1 Y0 + m) / rho mod n
// so a squaring is two products of H limbs and two reductions modulo n
// (4 H^2 multiply-adds), a product three and two (5 H^2), where the Montgomery
// product modulo n^2 of 2H limbs takes 8 H^2.  The digits are the p-adic
// digits of the residue, as in Hensel lifting; the two reductions are
// Montgomery's (Math. Comp. 44, 1985).
//
// An instance is a group of 2 TC lanes: TC lanes (chain 0) reduce X0 Y0, TC
// lanes (chain 1) reduce the rest, both with the same instructions; lane t of
// a chain holds limbs [t L, t L + L), H = TC L.  Limb i of m is added at limb i
// of chain 1 in step i, at no cost: it takes the place of a carry.  The one
// extra limb of rho keeps a result below n + 2^(32 H - 30), so no conditional
// subtraction is needed unless n's top limb is all ones; that case is handled
// behind one vote per pass.
//
// Multiplier limbs come from shared memory, [digit][limb][instance of the
// warp], multiplicands and running columns (mont.cuh) from registers.  n is
// any array of L words: registers, or with TC = 1 the kernel's constant bank,
// which frees L registers.
#pragma once
#include "mont.cuh"

namespace hg {

template <int TC, int L>
struct SqLanes {
  static constexpr int H = TC * L;
  static constexpr int IPW = 32 / (2 * TC);      // instances per warp
  static constexpr int kDigit = H * IPW + (IPW == 16 ? 16 : 0);  // words between the digits' areas
  static constexpr int kWords = 2 * kDigit;      // shared words per warp
  uint32_t lane, base, chain_base;  // warp lane; first lane of the group and of the chain
  int c, t, iw;                     // chain, lane in the chain, instance of the warp
  __device__ __forceinline__ SqLanes() {
    lane = threadIdx.x & 31u;
    iw = (int)(lane / (2 * TC));
    c = (int)(lane / TC) & 1;
    t = (int)(lane % TC);
    base = (uint32_t)iw * 2 * TC;
    chain_base = base + (uint32_t)c * TC;
  }
  // this lane's slice of digit d in the warp's area
  __device__ __forceinline__ uint32_t* limb(uint32_t* area, int d, int i) const {
    return area + d * kDigit + i * IPW + iw;
  }
};

// Write this lane's slice of its digit (digit 0 only if `both` is false).
template <int TC, int L>
__device__ __forceinline__ void sq_stage(uint32_t* area, const uint32_t (&x)[L], bool both, const SqLanes<TC, L>& g) {
  __syncwarp();
  if (both || g.c == 0) {
    uint32_t* s = g.limb(area, g.c, g.t * L);
#pragma unroll
    for (int j = 0; j < L; ++j) s[j * SqLanes<TC, L>::IPW] = x[j];
  }
  __syncwarp();
}

// Reduction of one limb in both chains, then the shift by one limb.  The
// pending c1 must be 0.  `in` enters the top limb of chain 0.
template <int TC, int L, class Mod>
__device__ __forceinline__ void sq_reduce_step(uint32_t (&Ev)[L], uint32_t (&Od)[L], uint32_t& ov, uint32_t& c1,
                                               const Mod& n, uint32_t np, uint32_t in, const SqLanes<TC, L>& g) {
  // both chains' lowest limbs travel together, so that chain 1 finds its m
  // (which depends on chain 0's) after one shuffle instead of two
  const uint32_t a = __shfl_sync(kFull, Ev[0], g.base);
  const uint32_t b = TC > 1 ? __shfl_sync(kFull, Ev[0], g.base + TC) : Ev[0];
  const uint32_t m0 = a * np;
  const uint32_t m = g.c ? (b + m0) * np : m0;
  const uint32_t inject = (g.c == 1 && g.t == 0) ? m0 : 0u;
  row_mac<L>(Ev, Od, ov, inject, n, m);
  uint32_t w = 0u;
  if constexpr (TC > 1) w = __shfl_down_sync(kFull, Ev[0], 1, TC);
  if (g.t == TC - 1) w = in;
  c1 = Ev[1];
#pragma unroll
  for (int j = 0; j + 2 < L; ++j) Ev[j] = Ev[j + 2];
  Ev[L - 2] = w;
  Ev[L - 1] = ov;
  ov = 0u;
}

// Columns -> limbs of both chains' results, below 2^(32 H).
template <int TC, int L, class Mod>
__device__ __forceinline__ void sq_settle(uint32_t (&x)[L], const uint32_t (&Ev)[L], const uint32_t (&Od)[L],
                                          uint32_t c1, const Mod& n, const SqLanes<TC, L>& g) {
  uint32_t top;
  if constexpr (TC == 1) {
    x[0] = add_cc(Ev[0], c1);
#pragma unroll
    for (int j = 1; j < L; ++j) x[j] = addc_cc(Ev[j], Od[j - 1]);
    top = addc(Od[L - 1], 0u);
  } else {
    const Group<TC> cg;
    top = settle<TC, L>(x, Ev, Od, 0u, c1, cg);
  }
  if (__any_sync(kFull, top != 0u)) {
    // a result at or above 2^(32 H): subtract n; X0 - n owes 1 to digit 1
    // (which is at least 1 there: m > 0 wherever digit 0 overflows)
    const uint32_t owed = __shfl_sync(kFull, top, g.base);
    uint32_t d[L], small[L];
#pragma unroll
    for (int j = 0; j < L; ++j) {
      d[j] = top ? n[j] : 0u;
      small[j] = 0u;
    }
    if (g.c == 1 && g.t == 0 && owed) small[0] = 1u;
    if constexpr (TC == 1) {
      x[0] = sub_cc(x[0], d[0]);
#pragma unroll
      for (int j = 1; j < L; ++j) x[j] = subc_cc(x[j], d[j]);
      (void)subc(0u, 0u);
      x[0] = sub_cc(x[0], small[0]);
#pragma unroll
      for (int j = 1; j < L; ++j) x[j] = subc_cc(x[j], 0u);
      (void)subc(0u, 0u);
    } else {
      const Group<TC> cg;
      (void)sub_full<TC, L>(x, x, d, cg);
      (void)sub_full<TC, L>(x, x, small, cg);
    }
  }
}

// Steps per round of a pass.  Between rounds the columns return to their
// registers (about two moves per limb, some of them on the multiply-add pipe),
// so more steps cost less, until the passes of a kernel leave the instruction
// cache: 131,072 CRT decryptions of 2048 bits with one 32-limb lane per chain
// took 170.5, 168.8 and 191 ms at 4, 8 and 16 steps, 19,456 of 3072 bits (48
// limbs) 85.0, 81.9 and 80.5 ms, 65,536 of 2048 bits with 16 limbs a lane 97.4,
// 91.0 and 87.7 ms.
template <int TC, int L>
constexpr int kSqUnroll = TC == 1 && L == 32 ? 8 : 16;

// z = (x * y [+ x2 * y2]) / rho in both chains, chain 0's m entering chain 1.
// y: this lane's multiplier limbs in shared memory (limb 0), doubled when
// `dbl` is 1.  kTwo adds the second product row.  z may alias x.
//   square:           x = own digit, y = digit 0, dbl = chain
//   product with Y:   x = Y's digit of the chain, y = X0, x2 = Y0, y2 = X1 (chain 1)
//   times integer Y0: x = Y0, y = own digit of X
template <int TC, int L, bool kTwo, class Mod>
__device__ __forceinline__ void sq_pass(uint32_t (&z)[L], const uint32_t (&x)[L], const uint32_t* y, uint32_t dbl,
                                        const uint32_t (&x2)[L], const uint32_t* y2, const Mod& n, uint32_t np,
                                        const SqLanes<TC, L>& g) {
  constexpr int H = TC * L, IPW = SqLanes<TC, L>::IPW, kU = kSqUnroll<TC, L>;
  static_assert(H % kU == 0 && kU % 2 == 0, "unrolling");
  uint32_t E[L], O[L];
#pragma unroll
  for (int j = 0; j < L; ++j) E[j] = O[j] = 0u;
  uint32_t ov = 0u, c1 = 0u, prev = 0u;
#pragma unroll 1
  for (int i = 0; i < H; i += kU) {
#pragma unroll
    for (int k = 0; k < kU; k += 2) {
      const uint32_t ya = y[(i + k) * IPW], yb = y[(i + k + 1) * IPW];
      row_mac<L>(E, O, ov, c1, x, __funnelshift_l(prev, ya, dbl));
      if constexpr (kTwo) row_mac<L>(E, O, ov, 0u, x2, g.c ? y2[(i + k) * IPW] : 0u);
      sq_reduce_step<TC, L>(E, O, ov, c1, n, np, 0u, g);
      row_mac<L>(O, E, ov, c1, x, __funnelshift_l(ya, yb, dbl));
      if constexpr (kTwo) row_mac<L>(O, E, ov, 0u, x2, g.c ? y2[(i + k + 1) * IPW] : 0u);
      sq_reduce_step<TC, L>(O, E, ov, c1, n, np, 0u, g);
      prev = yb;
    }
  }
  // the extra limb of rho: a doubled multiplier's top bit, or no product
  row_mac<L>(E, O, ov, c1, x, __funnelshift_l(prev, 0u, dbl));
  sq_reduce_step<TC, L>(E, O, ov, c1, n, np, 0u, g);
  sq_settle<TC, L>(z, O, E, c1, n, g);
}

// One reduction step without a product row.
template <int TC, int L, class Mod>
__device__ __forceinline__ void sq_redc_step(uint32_t (&Ev)[L], uint32_t (&Od)[L], uint32_t& ov, uint32_t& c1,
                                             const Mod& n, uint32_t np, uint32_t in, const SqLanes<TC, L>& g) {
  Ev[0] = add_cc(Ev[0], c1);
#pragma unroll
  for (int j = 0; j < L; ++j) Od[j] = addc_cc(Od[j], 0u);
  ov = addc(ov, 0u);
  c1 = 0u;
  sq_reduce_step<TC, L>(Ev, Od, ov, c1, n, np, in, g);
}

// Digits of W * 2^(-32 (kWide - H + 1)) for a raw number W of kWide >= H
// limbs (`src`, 16-byte aligned, this instance's): chain 0 takes the limbs in
// from below its top as it reduces.  kWide = H: a reduction of W by rho.
template <int TC, int L, int kWide, class Mod>
__device__ __forceinline__ void sq_from_raw(uint32_t (&z)[L], const uint32_t* __restrict__ src, const Mod& n,
                                            uint32_t np, const SqLanes<TC, L>& g) {
  constexpr int H = TC * L, kIn = kWide - H;
  static_assert(kIn % 4 == 0, "limbs");
  uint32_t E[L], O[L];
#pragma unroll
  for (int j = 0; j < L; ++j) {
    E[j] = g.c == 0 ? src[g.t * L + j] : 0u;
    O[j] = 0u;
  }
  uint32_t ov = 0u, c1 = 0u;
  const bool taker = g.c == 0 && g.t == TC - 1;
  const uint4* q = reinterpret_cast<const uint4*>(src + H);
  uint4 v = taker ? q[0] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
  for (int i = 0; i < kIn; i += 4) {
    const uint4 nx = (taker && i + 4 < kIn) ? q[i / 4 + 1] : make_uint4(0u, 0u, 0u, 0u);
    sq_redc_step<TC, L>(E, O, ov, c1, n, np, v.x, g);
    sq_redc_step<TC, L>(O, E, ov, c1, n, np, v.y, g);
    sq_redc_step<TC, L>(E, O, ov, c1, n, np, v.z, g);
    sq_redc_step<TC, L>(O, E, ov, c1, n, np, v.w, g);
    v = nx;
  }
  sq_redc_step<TC, L>(E, O, ov, c1, n, np, 0u, g);
  sq_settle<TC, L>(z, O, E, c1, n, g);
}

// z = x / rho (both digits): out of the Montgomery form.
template <int TC, int L, class Mod>
__device__ __forceinline__ void sq_redc(uint32_t (&z)[L], const uint32_t (&x)[L], const Mod& n, uint32_t np,
                                        const SqLanes<TC, L>& g) {
  constexpr int H = TC * L;
  uint32_t E[L], O[L];
#pragma unroll
  for (int j = 0; j < L; ++j) {
    E[j] = x[j];
    O[j] = 0u;
  }
  uint32_t ov = 0u, c1 = 0u;
#pragma unroll 1
  for (int i = 0; i < H; i += 2) {
    sq_redc_step<TC, L>(E, O, ov, c1, n, np, 0u, g);
    sq_redc_step<TC, L>(O, E, ov, c1, n, np, 0u, g);
  }
  sq_redc_step<TC, L>(E, O, ov, c1, n, np, 0u, g);
  sq_settle<TC, L>(z, O, E, c1, n, g);
}

}  // namespace hg
