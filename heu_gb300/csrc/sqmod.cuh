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
// Multiplier limbs come from shared memory in quads, [digit][limb / 4]
// [instance of the warp][4], so one 16-byte load feeds four steps;
// multiplicands and running columns (mont.cuh) are in registers.  n is any
// array of L words: registers, or with TC = 1 the kernel's constant bank,
// which frees L registers.
#pragma once
#include <type_traits>

#include "mont.cuh"

// Limbs a loop body of a pass takes (kSqUnroll); 0: by layout.  A unit that wants
// another number (batch_v0.cu) gets its passes, and all that is built from them,
// under names of their own.
#ifndef HG_SQ_UNROLL
#define HG_SQ_UNROLL 0
#endif
#define HG_SQ_JOIN_(a, b) a##b
#define HG_SQ_JOIN(a, b) HG_SQ_JOIN_(a, b)
#define HG_SQ_SPACE HG_SQ_JOIN(sq_unroll_, HG_SQ_UNROLL)

namespace hg {
inline namespace HG_SQ_SPACE {

template <int TC, int L>
struct SqLanes {
  static constexpr int H = TC * L;
  static constexpr int IPW = 32 / (2 * TC);      // instances per warp
  static constexpr int kDigit = H * IPW;         // shared words per digit and warp
  static constexpr int kVec = L % 4 == 0 ? 4 : 2;  // words of a lane's vector accesses
  uint32_t lane, base;  // warp lane; the group's first lane
  int c, t, iw;                     // chain, lane in the chain, instance of the warp
  __device__ __forceinline__ SqLanes() {
    lane = threadIdx.x & 31u;
    iw = (int)(lane / (2 * TC));
    c = (int)(lane / TC) & 1;
    t = (int)(lane % TC);
    base = (uint32_t)iw * 2 * TC;
  }
  // limb i (a multiple of 4) of digit d of this lane's instance
  __device__ __forceinline__ uint32_t* limb(uint32_t* area, int d, int i) const {
    return area + d * kDigit + (i * IPW + iw * 4);
  }
  // word offset, from limb 0, of vector v of this lane's slice
  __device__ __forceinline__ int slice_at(int v) const {
    const int i = t * L + v * kVec;
    return (i >> 2) * 4 * IPW + (i & 3);
  }
};

// This lane's slice to and from a digit's area (`digit` points at its limb 0
// of the instance).
template <int TC, int L>
__device__ __forceinline__ void sq_put(uint32_t* digit, const uint32_t (&x)[L], const SqLanes<TC, L>& g) {
  constexpr int V = SqLanes<TC, L>::kVec;
#pragma unroll
  for (int v = 0; v < L / V; ++v) {
    uint32_t* p = digit + g.slice_at(v);
    if constexpr (V == 4)
      *reinterpret_cast<uint4*>(p) = make_uint4(x[4 * v], x[4 * v + 1], x[4 * v + 2], x[4 * v + 3]);
    else
      *reinterpret_cast<uint2*>(p) = make_uint2(x[2 * v], x[2 * v + 1]);
  }
}

template <int TC, int L>
__device__ __forceinline__ void sq_get(uint32_t (&x)[L], const uint32_t* digit, const SqLanes<TC, L>& g) {
  constexpr int V = SqLanes<TC, L>::kVec;
#pragma unroll
  for (int v = 0; v < L / V; ++v) {
    const uint32_t* p = digit + g.slice_at(v);
    if constexpr (V == 4) {
      const uint4 q = *reinterpret_cast<const uint4*>(p);
      x[4 * v] = q.x;
      x[4 * v + 1] = q.y;
      x[4 * v + 2] = q.z;
      x[4 * v + 3] = q.w;
    } else {
      const uint2 q = *reinterpret_cast<const uint2*>(p);
      x[2 * v] = q.x;
      x[2 * v + 1] = q.y;
    }
  }
}

// Write this lane's slice of its digit (digit 0 only if `both` is false).
template <int TC, int L>
__device__ __forceinline__ void sq_stage(uint32_t* area, const uint32_t (&x)[L], bool both, const SqLanes<TC, L>& g) {
  __syncwarp();
  if (both || g.c == 0) sq_put<TC, L>(g.limb(area, g.c, 0), x, g);
  __syncwarp();
}

// Reduction of one limb in both chains, then the shift by one limb.  The
// pending c1 must be 0.  `in` enters the top limb of chain 0.  Without kJoin
// the chains are two reductions modulo n of their own.  a, b: the lowest limbs
// of the instance's chains, which travel together so that chain 1 finds its m
// (it depends on chain 0's) after one shuffle's time and not two.
template <int TC, int L, bool kJoin, class Mod>
__device__ __forceinline__ void sq_reduce_with(uint32_t (&Ev)[L], uint32_t (&Od)[L], uint32_t& ov, uint32_t& c1,
                                               const Mod& n, uint32_t np, uint32_t in, uint32_t a, uint32_t b,
                                               const SqLanes<TC, L>& g) {
  const uint32_t m0 = a * np;
  const uint32_t m = g.c ? (kJoin ? b + m0 : b) * np : m0;
  row_mac<L>(Ev, Od, ov, (kJoin && g.c == 1 && g.t == 0) ? m0 : 0u, n, m);
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

template <int TC, int L, bool kJoin = true, class Mod>
__device__ __forceinline__ void sq_reduce_step(uint32_t (&Ev)[L], uint32_t (&Od)[L], uint32_t& ov, uint32_t& c1,
                                               const Mod& n, uint32_t np, uint32_t in, const SqLanes<TC, L>& g) {
  const uint32_t a = __shfl_sync(kFull, Ev[0], g.base);
  const uint32_t b = TC > 1 ? __shfl_sync(kFull, Ev[0], g.base + TC) : Ev[0];
  sq_reduce_with<TC, L, kJoin>(Ev, Od, ov, c1, n, np, in, a, b, g);
}

// One step of the layouts for few ciphertexts, where the chain of dependent
// instructions sets the time: `low` is this step's lowest limb in the chains'
// first lanes, found ahead of the rows, so its shuffle runs under the product
// rows; the next step's is Od[0] + Ev[1] after the reduction row plus `next`,
// the lowest limb of its products.
template <int TC, int L, bool kTwo, bool kJoin, class Mod>
__device__ __forceinline__ void sq_step_early(uint32_t (&Ev)[L], uint32_t (&Od)[L], uint32_t& ov, uint32_t& c1,
                                              uint32_t& low, uint32_t next, const uint32_t (&x)[L], uint32_t y,
                                              const uint32_t (&x2)[L], uint32_t y2, const Mod& n, uint32_t np,
                                              const SqLanes<TC, L>& g) {
  const uint32_t a = __shfl_sync(kFull, low, g.base);
  const uint32_t b = __shfl_sync(kFull, low, g.base + TC);
  row_mac<L>(Ev, Od, ov, c1, x, y);
  if constexpr (kTwo) row_mac<L>(Ev, Od, ov, 0u, x2, y2);
  sq_reduce_with<TC, L, kJoin>(Ev, Od, ov, c1, n, np, 0u, a, b, g);
  low = Od[0] + c1 + next;
}

// Columns -> limbs of both chains' results, below 2^(32 H).
template <int TC, int L, bool kJoin = true, class Mod>
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
    if (kJoin && g.c == 1 && g.t == 0 && owed) small[0] = 1u;
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
// 91.0 and 87.7 ms.  (Multipliers in 16-byte loads then took 1 to 3% off each.)
template <int TC, int L>
constexpr int kSqUnroll = HG_SQ_UNROLL ? HG_SQ_UNROLL : TC == 1 && L == 32 ? 8 : 16;

// Layouts whose passes run sq_step_early: the widest of the primes' lengths,
// which only few ciphertexts take.  8 CRT decryptions of 2048 bits (16 lanes a
// chain) took 1.92 ms without and 1.71 with it, 3072 bits (8 lanes) 5.20 and
// 4.90.  With 4 limbs a lane and more steps a pass it gains nothing (one
// encryption of 2048 bits 0.102 and 0.104 ms), and with several warps a
// scheduler its extra work costs 2 to 3%.
template <int TC, int L>
constexpr bool kSqEarly = L == 2 || (TC == 8 && L == 6);

// z = (x * y [+ x2 * y2]) / rho in both chains, chain 0's m entering chain 1.
// y: this lane's multiplier limbs in shared memory (limb 0), doubled when
// `dbl` is 1.  kTwo adds the second product row.  z may alias x.
//   square:           x = own digit, y = digit 0, dbl = chain
//   product with Y:   x = Y's digit of the chain, y = X0, x2 = Y0, y2 = X1 (chain 1)
//   times integer Y0: x = Y0, y = own digit of X
// kJoin = false: z_c = x_c * y_c / rho modulo n in each chain for itself.
// `ytop` is limb H of an undoubled multiplier: below 2^31 it leaves the result
// below n + x / 2, so the subtraction behind the vote brings it below 2^(32 H)
// and the caller's one more, x being less than 2 n, below n.  The encryption's is
// the top word of a sum of npos + 2 numbers, MatMul's that of its doubled sum,
// which launch_mm_planes holds below 2^31.
template <int TC, int L, bool kTwo, bool kJoin = true, class Mod>
__device__ __forceinline__ void sq_pass(uint32_t (&z)[L], const uint32_t (&x)[L], const uint32_t* y, uint32_t dbl,
                                        uint32_t ytop, const uint32_t (&x2)[L], const uint32_t* y2, const Mod& n,
                                        uint32_t np, const SqLanes<TC, L>& g) {
  constexpr int H = TC * L, IPW = SqLanes<TC, L>::IPW, kU = kSqUnroll<TC, L>;
  static_assert(H % kU == 0 && kU % 4 == 0, "unrolling");
  uint32_t E[L], O[L];
#pragma unroll
  for (int j = 0; j < L; ++j) E[j] = O[j] = 0u;
  uint32_t ov = 0u, c1 = 0u, prev = 0u;
  if constexpr ((kSqEarly<TC, L>)) {
    uint4 q = *reinterpret_cast<const uint4*>(y);
    uint4 q2 = kTwo ? *reinterpret_cast<const uint4*>(y2) : make_uint4(0u, 0u, 0u, 0u);
    if (kTwo && !g.c) q2 = make_uint4(0u, 0u, 0u, 0u);
    // the lowest limb of the products of multiplier limbs v (and w)
    auto lowest = [&](uint32_t v, uint32_t w) { return kTwo ? x[0] * v + x2[0] * w : x[0] * v; };
    uint32_t v0 = __funnelshift_l(0u, q.x, dbl);
    uint32_t low = lowest(v0, q2.x);
#pragma unroll 4
    for (int i = 0; i < H; i += 4) {
      const int at = i + 4 < H ? (i + 4) * IPW : 0;
      uint4 p = *reinterpret_cast<const uint4*>(y + at);
      uint4 p2 = kTwo ? *reinterpret_cast<const uint4*>(y2 + at) : make_uint4(0u, 0u, 0u, 0u);
      if (kTwo && !g.c) p2 = make_uint4(0u, 0u, 0u, 0u);
      if (i + 4 >= H) {
        p.x = ytop;
        p2.x = 0u;
      }
      const uint32_t v1 = __funnelshift_l(q.x, q.y, dbl), v2 = __funnelshift_l(q.y, q.z, dbl);
      const uint32_t v3 = __funnelshift_l(q.z, q.w, dbl), v4 = __funnelshift_l(q.w, p.x, dbl);
      sq_step_early<TC, L, kTwo, kJoin>(E, O, ov, c1, low, lowest(v1, q2.y), x, v0, x2, q2.x, n, np, g);
      sq_step_early<TC, L, kTwo, kJoin>(O, E, ov, c1, low, lowest(v2, q2.z), x, v1, x2, q2.y, n, np, g);
      sq_step_early<TC, L, kTwo, kJoin>(E, O, ov, c1, low, lowest(v3, q2.w), x, v2, x2, q2.z, n, np, g);
      sq_step_early<TC, L, kTwo, kJoin>(O, E, ov, c1, low, lowest(v4, p2.x), x, v3, x2, q2.w, n, np, g);
      v0 = v4;
      q = p;
      q2 = p2;
    }
    sq_step_early<TC, L, false, kJoin>(E, O, ov, c1, low, 0u, x, v0, x2, 0u, n, np, g);
  } else {
#pragma unroll 1
    for (int i = 0; i < H; i += kU) {
#pragma unroll
      for (int k = 0; k < kU; k += 4) {
        const uint4 q = *reinterpret_cast<const uint4*>(y + (i + k) * IPW);
        const uint4 q2 = kTwo ? *reinterpret_cast<const uint4*>(y2 + (i + k) * IPW) : make_uint4(0u, 0u, 0u, 0u);
        row_mac<L>(E, O, ov, c1, x, __funnelshift_l(prev, q.x, dbl));
        if constexpr (kTwo) row_mac<L>(E, O, ov, 0u, x2, g.c ? q2.x : 0u);
        sq_reduce_step<TC, L, kJoin>(E, O, ov, c1, n, np, 0u, g);
        row_mac<L>(O, E, ov, c1, x, __funnelshift_l(q.x, q.y, dbl));
        if constexpr (kTwo) row_mac<L>(O, E, ov, 0u, x2, g.c ? q2.y : 0u);
        sq_reduce_step<TC, L, kJoin>(O, E, ov, c1, n, np, 0u, g);
        row_mac<L>(E, O, ov, c1, x, __funnelshift_l(q.y, q.z, dbl));
        if constexpr (kTwo) row_mac<L>(E, O, ov, 0u, x2, g.c ? q2.z : 0u);
        sq_reduce_step<TC, L, kJoin>(E, O, ov, c1, n, np, 0u, g);
        row_mac<L>(O, E, ov, c1, x, __funnelshift_l(q.z, q.w, dbl));
        if constexpr (kTwo) row_mac<L>(O, E, ov, 0u, x2, g.c ? q2.w : 0u);
        sq_reduce_step<TC, L, kJoin>(O, E, ov, c1, n, np, 0u, g);
        prev = q.w;
      }
    }
    // the extra limb of rho: a doubled multiplier's top bit, or ytop
    row_mac<L>(E, O, ov, c1, x, __funnelshift_l(prev, ytop, dbl));
    sq_reduce_step<TC, L, kJoin>(E, O, ov, c1, n, np, 0u, g);
  }
  sq_settle<TC, L, kJoin>(z, O, E, c1, n, g);
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
// limbs (`src`, this instance's; a caller's array, of which no more than 8-byte
// alignment is asked): chain 0 takes the limbs in from below its top as it
// reduces.  kWide = H: a reduction of W by rho.
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
  auto limbs = [&](int i) {
    const uint2* q = reinterpret_cast<const uint2*>(src + H + i);
    const uint2 lo = q[0], hi = q[1];
    return make_uint4(lo.x, lo.y, hi.x, hi.y);
  };
  uint4 v = taker ? limbs(0) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
  for (int i = 0; i < kIn; i += 4) {
    const uint4 nx = (taker && i + 4 < kIn) ? limbs(i + 4) : make_uint4(0u, 0u, 0u, 0u);
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

// ---- tables of a warp in global scratch ---------------------------------------
// Vector words of a lane's slice.
template <int L>
struct SliceVec {
  using T = typename std::conditional<L % 4 == 0, uint4, uint2>::type;
  static constexpr int kN = L % 4 == 0 ? L / 4 : L / 2;
};

// A warp's table: [entry][vector][lane], so the load or store of one entry by
// all lanes is one contiguous run.
template <int L>
__device__ __forceinline__ void table_load(uint32_t (&x)[L], const uint32_t* tb, int e, uint32_t lane) {
  using V = typename SliceVec<L>::T;
  constexpr int kN = SliceVec<L>::kN, kW = sizeof(V) / 4;
  const V* p = reinterpret_cast<const V*>(tb) + (size_t)e * kN * 32 + lane;
#pragma unroll
  for (int q = 0; q < kN; ++q) {
    const V v = p[q * 32];
    x[kW * q] = v.x;
    x[kW * q + 1] = v.y;
    if constexpr (kW == 4) {
      x[kW * q + 2] = v.z;
      x[kW * q + 3] = v.w;
    }
  }
}

template <int L>
__device__ __forceinline__ void table_store(uint32_t* tb, int e, uint32_t lane, const uint32_t (&x)[L]) {
  using V = typename SliceVec<L>::T;
  constexpr int kN = SliceVec<L>::kN, kW = sizeof(V) / 4;
  V* p = reinterpret_cast<V*>(tb) + (size_t)e * kN * 32 + lane;
#pragma unroll
  for (int q = 0; q < kN; ++q) {
    if constexpr (kW == 4)
      p[q * 32] = make_uint4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
    else
      p[q * 32] = make_uint2(x[2 * q], x[2 * q + 1]);
  }
}

// ---- digit helpers over one chain -------------------------------------------
// r = a + b over the chain's H limbs; returns the carry out (in every lane).
template <int TC, int L>
__device__ __forceinline__ uint32_t chain_add(uint32_t (&r)[L], const uint32_t (&a)[L], const uint32_t (&b)[L]) {
  if constexpr (TC == 1) {
    r[0] = add_cc(a[0], b[0]);
#pragma unroll
    for (int j = 1; j < L; ++j) r[j] = addc_cc(a[j], b[j]);
    return addc(0u, 0u);
  } else {
    const Group<TC> cg;
    return add_full<TC, L>(r, a, b, cg);
  }
}

// r = a - b; returns the borrow out.
template <int TC, int L>
__device__ __forceinline__ uint32_t chain_sub(uint32_t (&r)[L], const uint32_t (&a)[L], const uint32_t (&b)[L]) {
  if constexpr (TC == 1) {
    r[0] = sub_cc(a[0], b[0]);
#pragma unroll
    for (int j = 1; j < L; ++j) r[j] = subc_cc(a[j], b[j]);
    return subc(0u, 0u) & 1u;
  } else {
    const Group<TC> cg;
    return sub_full<TC, L>(r, a, b, cg);
  }
}

// x (with `top` above its limbs) less n where that is not negative.
template <int TC, int L>
__device__ __forceinline__ void chain_reduce_once(uint32_t (&x)[L], uint32_t top, const uint32_t (&n)[L]) {
  uint32_t d[L];
  const uint32_t borrow = chain_sub<TC, L>(d, x, n);
  select_slice<L>(x, top != 0u || borrow == 0u, d, x);
}

// Limbs plus a carry word per lane -> limbs; returns the word above the top.
template <int TC, int L>
__device__ __forceinline__ uint32_t chain_settle(uint32_t (&x)[L], uint32_t carry) {
  if constexpr (TC == 1) {
    return carry;
  } else {
    const Group<TC> cg;
    uint32_t c[L];
    c[0] = __shfl_up_sync(kFull, carry, 1, TC);
    if (cg.t == 0) c[0] = 0u;
#pragma unroll
    for (int j = 1; j < L; ++j) c[j] = 0u;
    const uint32_t out = add_full<TC, L>(x, x, c, cg);
    return __shfl_sync(kFull, carry, TC - 1, TC) + out;
  }
}

// Is the raw number of 2 TC * W limbs at `a` below the one at `b`?
template <int TC, int W>
__device__ __forceinline__ bool raw_below(const uint32_t* __restrict__ a, const uint32_t* __restrict__ b) {
  const Group<2 * TC> g;
  a += g.t * W;
  b += g.t * W;
  uint32_t borrow = 0u;
  bool same = true;
#pragma unroll 4
  for (int j = 0; j < W; ++j) {
    const uint64_t d = (uint64_t)a[j] - b[j] - borrow;
    borrow = (uint32_t)(d >> 63);
    same = same && a[j] == b[j];
  }
  uint32_t out;
  (void)lookahead<2 * TC>(g, borrow != 0u, same, 0u, out);
  return out != 0u;
}

// The residue x / rho as a raw number below n^2: chain c gets limbs
// [c H + t L, c H + t L + L) of it.  `area` holds two digits.
//   x / rho = x0 - x1 n with 0 <= x0 <= n, 0 <= x1 <= n + 1, and then
//   x0 + (n - x1) n with both digits in [0, n).
template <int TC, int L, class Mod>
__device__ __forceinline__ void sq_to_raw(uint32_t (&r)[L], const uint32_t (&xin)[L], uint32_t* area, const Mod& n,
                                          uint32_t np, const SqLanes<TC, L>& g) {
  constexpr int H = TC * L, IPW = SqLanes<TC, L>::IPW;
  uint32_t x[L], v[L], nn[L], d[L];
  sq_redc<TC, L>(x, xin, n, np, g);
#pragma unroll
  for (int j = 0; j < L; ++j) nn[j] = n[j];
  // both digits below n; x0 = n is 0 and owes 1 to digit 1
  const bool whole = chain_sub<TC, L>(d, x, nn) == 0u;
  const bool owed = __shfl_sync(kFull, (int)whole, g.base) != 0;
  select_slice<L>(x, whole, d, x);
  // v = n - x1 + owed mod n (chain 1)
  (void)chain_sub<TC, L>(v, nn, x);
#pragma unroll
  for (int j = 0; j < L; ++j) d[j] = 0u;
  if (g.t == 0 && owed) d[0] = 1u;
  const uint32_t top = chain_add<TC, L>(v, v, d);
  chain_reduce_once<TC, L>(v, top, nn);
  __syncwarp();
  if (g.c == 1) sq_put<TC, L>(g.limb(area, 1, 0), v, g);
  __syncwarp();
  // x0 + v n: rows of n, the lowest limb leaves in every step
  const uint32_t* y = g.limb(area, 1, 0);
  uint32_t* low = g.limb(area, 0, 0);
  uint32_t E[L], O[L], ov = 0u, c1 = 0u;
#pragma unroll
  for (int j = 0; j < L; ++j) {
    E[j] = x[j];
    O[j] = 0u;
  }
  auto step = [&](uint32_t (&Ev)[L], uint32_t (&Od)[L], uint32_t w) {
    row_mac<L>(Ev, Od, ov, c1, nn, w);
    const uint32_t out = Ev[0];
    if constexpr (TC == 1) {
      c1 = Ev[1];
#pragma unroll
      for (int j = 0; j + 2 < L; ++j) Ev[j] = Ev[j + 2];
      Ev[L - 2] = 0u;
      Ev[L - 1] = ov;
      ov = 0u;
    } else {
      const Group<TC> cg;
      shift_limb<TC, L>(Ev, ov, c1, cg);
    }
    return out;
  };
#pragma unroll 1
  for (int i = 0; i < H; i += 4) {
    const uint4 q = *reinterpret_cast<const uint4*>(y + i * IPW);
    uint4 o;
    o.x = step(E, O, q.x);
    o.y = step(O, E, q.y);
    o.z = step(E, O, q.z);
    o.w = step(O, E, q.w);
    if (g.c == 0 && g.t == 0) *reinterpret_cast<uint4*>(low + i * IPW) = o;
  }
  if constexpr (TC == 1) {
    x[0] = add_cc(E[0], c1);
#pragma unroll
    for (int j = 1; j < L; ++j) x[j] = addc_cc(E[j], O[j - 1]);
    (void)addc(0u, 0u);
  } else {
    const Group<TC> cg;
    (void)settle<TC, L>(x, E, O, ov, c1, cg);
  }
  __syncwarp();
  sq_get<TC, L>(r, low, g);
#pragma unroll
  for (int j = 0; j < L; ++j) {
    const uint32_t h = __shfl_sync(kFull, x[j], g.c ? g.lane - TC : g.lane);
    r[j] = g.c ? h : r[j];
  }
}

}  // namespace HG_SQ_SPACE
}  // namespace hg
