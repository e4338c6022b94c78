// Mul(ct, k) for 64-bit k in two digits to the base n (sqmod.cuh): c^|k| mod
// n^2 by windows at fixed places, so that all instances of a warp square and
// multiply in the same steps (a squaring costs 4 H^2 multiply-adds, a product
// 6, a step in which some instance multiplies would cost 6 for all).  k = 0
// gives the Montgomery identity (evaluator.cc:105-106); k < 0 is finished by a
// batch inverse afterwards (evaluator.cc:119-121).
#pragma once
#include "paillier_ops.cuh"
#include "sqmod.cuh"

namespace hg {
inline namespace HG_SQ_SPACE {

// `tb`: mul_slots(wm) entries of this warp, `area`: two digits.
template <int TC, int L, class Mod>
__device__ __forceinline__ void sq_mul(const Mod& n, const KeyConst& kc, const uint32_t* __restrict__ a,
                                       const int64_t* __restrict__ kk, uint32_t* __restrict__ out, size_t i,
                                       bool active, uint32_t* tb, int wm, uint32_t* area, uint32_t* err,
                                       const SqLanes<TC, L>& g) {
  constexpr int H = TC * L, S = 2 * H;
  const uint32_t np = kc.npn;
  const int ntab = 1 << wm;
  const uint64_t e = abs_i64(kk[i]);
  const bool ok = raw_below<TC, L>(a + i * S, kc.N);
  if (active && !ok && g.lane == g.base) atomicOr(err, kErrCtRange);
  uint32_t x[L];
  auto put_const = [&](const uint32_t* c, int slot) {
    load_slice<L>(x, c + g.c * H + g.t * L);
    table_store<L>(tb, slot, g.lane, x);
  };
  put_const(kc.one, 0);
  put_const(kc.kin, ntab);
  put_const(kc.kout, ntab + 1);
  // windows of the warp's longest scalar
  const int bits = (int)__reduce_max_sync(kFull, (unsigned)(64 - __clzll((long long)e)));
  const int wins = max(1, (bits + wm - 1) / wm);
  auto digit = [&](int w) { return (int)((e >> (w * wm)) & (uint64_t)(ntab - 1)); };
  sq_from_raw<TC, L, S>(x, a + i * S, n, np, g);
  // one loop, so that each kind of pass is compiled once: into the form (step
  // 0), the powers (steps up to ntab - 2), the windows, out of the form
  const int steps = ntab + (wins - 1) * (wm + 1);
#pragma unroll 1
  for (int s = 0; s < steps; ++s) {
    int slot = -1, keep = -1;  // multiply by the slot's entry (-1: square); store to
    if (s == 0) {
      slot = ntab;
      keep = 1;
    } else if (s < ntab - 1) {
      keep = s + 1;
      if (keep & 1)
        slot = 1;
      else
        table_load<L>(x, tb, keep >> 1, g.lane);
    } else {
      if (s == ntab - 1) table_load<L>(x, tb, digit(wins - 1), g.lane);
      const int q = s - (ntab - 1), w = q / (wm + 1);
      if (s == steps - 1)
        slot = ntab + 1;
      else if (q - w * (wm + 1) == wm)
        slot = digit(wins - 2 - w);
    }
    const bool product = __any_sync(kFull, slot >= 0);
    sq_stage<TC, L>(area, x, product, g);
    if (!product) {
      sq_pass<TC, L, false>(x, x, g.limb(area, 0, 0), (uint32_t)g.c, 0u, x, nullptr, n, np, g);
    } else {
      uint32_t y0[L];
      table_load<L>(x, tb, slot, g.lane);
      table_load<L>(y0, tb, slot, g.lane - g.c * TC);
      sq_pass<TC, L, true>(x, x, g.limb(area, 0, 0), 0u, 0u, y0, g.limb(area, 1, 0), n, np, g);
    }
    if (keep >= 0) table_store<L>(tb, keep, g.lane, x);
  }
  uint32_t r[L];
  sq_to_raw<TC, L>(r, x, area, n, np, g);
  if (active) store_slice<L>(out + i * S + g.c * H + g.t * L, r);
}

}  // namespace HG_SQ_SPACE
}  // namespace hg
