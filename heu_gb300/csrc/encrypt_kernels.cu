// Fixed-base encryption of ZPaillier keys and the tables it reads
// (sq_encrypt.cuh).  OU keys, whose modulus is no square, encrypt with
// k_encrypt (paillier_kernels.cu).
#include <algorithm>
#include <atomic>
#include <cmath>

#include "sq_encrypt.cuh"

namespace hg {

namespace {

template <int H>
struct Modulus {
  uint32_t n[H];
};

// A warp per group of ciphertexts, or kWarps warps of each of kBlocks blocks
// (a cluster) that share its products.
//
// Bound: the fmaheavy pipe.  131,072 encryptions of 2048 bits at table window
// 16 took 32.2 ms as 66 products modulo n^2 each; as 63 products by integers of
// n's length and a tail of about 7 they take 17.4 ms.
template <int TC, int L, int kWarps, int kBlocks = 1>
__global__ void __launch_bounds__(32 * kWarps)
    k_sq_encrypt(const __grid_constant__ Modulus<TC * L> mod, const __grid_constant__ KeyConst kc,
                 const __grid_constant__ EncArgs a, uint32_t* __restrict__ out, size_t count, uint32_t* err) {
  using G = SqLanes<TC, L>;
  extern __shared__ __align__(16) uint32_t enc_area[];
  const G g;
  const size_t inst = (size_t)(blockIdx.x / kBlocks) * G::IPW + g.iw;
  const bool active = inst < count;
  const size_t i = active ? inst : count - 1;
  uint32_t* area = enc_area + (threadIdx.x >> 5) * kEncWords<TC, L>;
  uint32_t* carries = enc_area + kWarps * kEncWords<TC, L>;
  if constexpr (TC == 1) {
    sq_encrypt<TC, L, kWarps, kBlocks>(mod.n, kc, a, out, i, active, area, carries, err, g);
  } else {
    uint32_t n[L];
    load_slice<L>(n, kc.n + g.t * L);
    sq_encrypt<TC, L, kWarps, kBlocks>(n, kc, a, out, i, active, area, carries, err, g);
  }
}

template <int TC, int L, int kWarps>
constexpr size_t enc_smem() {
  return (size_t)(kWarps * kEncWords<TC, L> + (kWarps > 1 ? kWarps * 32 : 0)) * 4;
}

// Layouts by (limbs of n, log2 of the lanes per chain).
#define HG_DISPATCH_SQ(H, LOGTC, ...)                                           \
  switch ((H) * 8 + (LOGTC)) {                                                  \
    case 256: { constexpr int TC = 1, L = 32; __VA_ARGS__; } break;             \
    case 257: { constexpr int TC = 2, L = 16; __VA_ARGS__; } break;             \
    case 258: { constexpr int TC = 4, L = 8; __VA_ARGS__; } break;              \
    case 260: { constexpr int TC = 16, L = 2; __VA_ARGS__; } break;             \
    case 513: { constexpr int TC = 2, L = 32; __VA_ARGS__; } break;             \
    case 514: { constexpr int TC = 4, L = 16; __VA_ARGS__; } break;             \
    case 515: { constexpr int TC = 8, L = 8; __VA_ARGS__; } break;              \
    case 516: { constexpr int TC = 16, L = 4; __VA_ARGS__; } break;             \
    case 769: { constexpr int TC = 2, L = 48; __VA_ARGS__; } break;             \
    case 770: { constexpr int TC = 4, L = 24; __VA_ARGS__; } break;             \
    case 771: { constexpr int TC = 8, L = 12; __VA_ARGS__; } break;             \
    case 772: { constexpr int TC = 16, L = 6; __VA_ARGS__; } break;             \
    default: return cudaErrorInvalidValue;                                      \
  }
#define HG_DISPATCH_SQ16(H, ...)                                                \
  switch (H) {                                                                  \
    case 32: { constexpr int TC = 16, L = 2; __VA_ARGS__; } break;              \
    case 64: { constexpr int TC = 16, L = 4; __VA_ARGS__; } break;              \
    case 96: { constexpr int TC = 16, L = 6; __VA_ARGS__; } break;              \
    default: return cudaErrorInvalidValue;                                      \
  }

constexpr int kShareWarps = 8;
constexpr int kClusterWarps = 4;  // a warp for each scheduler

template <int TC, int L, int kBlocks>
cudaError_t launch_cluster(const Modulus<TC * L>& m, const KeyConst& kc, const EncArgs& a, uint32_t* out, size_t count,
                           uint32_t* err, cudaStream_t st) {
  cudaLaunchAttribute at{};
  at.id = cudaLaunchAttributeClusterDimension;
  at.val.clusterDim.x = kBlocks;
  at.val.clusterDim.y = at.val.clusterDim.z = 1;
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)count * kBlocks);
  cfg.blockDim = dim3(32 * kClusterWarps);
  cfg.dynamicSmemBytes = enc_smem<TC, L, kClusterWarps>();
  cfg.stream = st;
  cfg.attrs = &at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, k_sq_encrypt<TC, L, kClusterWarps, kBlocks>, m, kc, a, out, count, err);
}

// ---------------------------------------------------------------------------
// tables
// ---------------------------------------------------------------------------
// bases[pos] = digits X0 | X1 of h^(2^(w pos)) rho and rho^2 / X0 mod n (3 H
// limbs): warp 0 squares the digits, warp 1 the inverse.
template <int TC, int L>
__global__ void __launch_bounds__(64) k_sq_bases(const __grid_constant__ KeyConst kc,
                                                 const uint32_t* __restrict__ first, uint32_t* __restrict__ bases) {
  using G = SqLanes<TC, L>;
  constexpr int H = G::H;
  __shared__ __align__(16) uint32_t areas[2][2 * G::kDigit];
  const G g;
  const int warp = threadIdx.x >> 5;
  uint32_t* area = areas[warp];
  uint32_t n[L], x[L];
  load_slice<L>(n, kc.n + g.t * L);
  load_slice<L>(x, first + (warp ? 2 * H : g.c * H) + g.t * L);
#pragma unroll 1
  for (int pos = 0; pos < kc.npos; ++pos) {
    if (g.iw == 0 && (warp == 0 || g.c == 0))
      store_slice<L>(bases + (size_t)pos * 3 * H + (warp ? 2 * H : g.c * H) + g.t * L, x);
#pragma unroll 1
    for (int s = 0; s < kc.w; ++s) {
      sq_stage<TC, L>(area, x, false, g);
      if (warp == 0)
        sq_pass<TC, L, false>(x, x, g.limb(area, 0, 0), (uint32_t)g.c, 0u, x, nullptr, n, kc.npn, g);
      else
        sq_pass<TC, L, false, false>(x, x, g.limb(area, 0, 0), 0u, 0u, x, nullptr, n, kc.npn, g);
    }
  }
}

// Entries of positions [pos0, pos0 + npos): level < 0 makes entry d = 1 from
// the bases, level j >= 0 entries d in [2^j + 1, min(2^(j+1), 2^w - 1)] as
// entry(2^j) * entry(d - 2^j); level w multiplies every entry by that of the
// output's radix (position 0, at the end).  inv[(pos - pos0) * ent + d - 1]
// holds rho^2 / Y0 mod n of the entries so far.  A group makes two entries: the
// products Y0 Y0' one after the other (both chains), then the inverses and
// y = Z1 / Z0 + y_a + y_b of both at once, one per chain; 8 H^2 multiply-adds
// an entry, as a product modulo n^2 takes.
template <int TC, int L>
__global__ void __launch_bounds__(128) k_sq_level(const __grid_constant__ KeyConst kc, uint32_t* __restrict__ table,
                                                  uint32_t* __restrict__ inv, const uint32_t* __restrict__ bases,
                                                  int pos0, size_t npos, int level, int subset) {
  using G = SqLanes<TC, L>;
  constexpr int H = G::H, S = 2 * H;
  __shared__ __align__(16) uint32_t areas[4][4 * G::kDigit];
  const G g;
  uint32_t* area = areas[threadIdx.x >> 5];
  uint32_t* area2 = area + 2 * G::kDigit;
  const size_t ent = (size_t)((1u << kc.w) - 1u);
  const bool scale = level == kc.w;
  const size_t lo = level < 0 || scale ? 1 : (1ull << level) + 1ull;
  const size_t hi = level < 0 ? 1 : scale ? ent : min((size_t)(1ull << (level + 1)) - (subset ? 1 : 0), ent);
  if (hi < lo) return;
  const size_t per = hi - lo + 1, total = per * npos;
  const size_t pair = ((size_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * G::IPW;
  if (2 * pair >= total) return;
  // this group's two entries; past the end the last one again
  auto place = [&](int k, size_t& p, size_t& d) {
    const size_t u = min(2 * (pair + g.iw) + (size_t)k, total - 1);
    p = u / per;
    d = lo + u % per;
  };
  size_t p, d;
  place(g.c, p, d);
  uint32_t n[L], x[L], z[L], y[L];
  load_slice<L>(n, kc.n + g.t * L);
  const size_t half = level < 0 || scale ? 0 : (size_t)1 << level;
  // the factors of entry d of (relative) position p, and their inverses
  auto left = [&](size_t p, size_t d) { return table + ((size_t)(pos0 + p) * ent + (scale ? d : half) - 1) * S; };
  auto right = [&](size_t p, size_t d) -> const uint32_t* {
    return scale ? kc.e0 : table + ((size_t)(pos0 + p) * ent + d - half - 1) * S;
  };
  if (level < 0) {
    // y = X1 / X0 times rho
    const uint32_t* b = bases + (size_t)(pos0 + p) * 3 * H + g.t * L;
    load_slice<L>(x, b + H);
    if (g.c == 1) sq_put<TC, L>(g.limb(area, 1, 0), x, g);
    if (g.c == 0) sq_put<TC, L>(g.limb(area, 0, 0), x, g);
    __syncwarp();
    load_slice<L>(x, b + 2 * H);
    store_slice<L>(inv + p * ent * H + g.t * L, x);
    sq_pass<TC, L, false, false>(y, x, g.limb(area, g.c, 0), 0u, 0u, x, nullptr, n, kc.npn, g);
    load_slice<L>(x, b);
  } else {
#pragma unroll 1
    for (int k = 0; k < 2; ++k) {
      size_t pk, dk;
      place(k, pk, dk);
      load_slice<L>(x, right(pk, dk) + g.t * L);
      __syncwarp();
      if (g.c == 0) sq_put<TC, L>(g.limb(area2, 0, 0), x, g);
      __syncwarp();
      load_slice<L>(x, left(pk, dk) + g.t * L);
      if (g.c == 1) {
#pragma unroll
        for (int j = 0; j < L; ++j) x[j] = 0u;
      }
      sq_pass<TC, L, false>(z, x, g.limb(area2, 0, 0), 0u, 0u, x, nullptr, n, kc.npn, g);
      // chain k keeps Z0 of entry k; Z1 waits as its multiplier
      if (g.c == 1) sq_put<TC, L>(g.limb(area, k, 0), z, g);
#pragma unroll
      for (int j = 0; j < L; ++j) {
        const uint32_t v = __shfl_sync(kFull, z[j], g.base + g.t);
        y[j] = (g.c == k) ? v : y[j];
      }
    }
    // inverses, one entry per chain
    const uint32_t* irow = inv + p * ent * H + g.t * L;
    load_slice<L>(x, scale ? kc.ie0 + g.t * L : irow + (d - half - 1) * H);
    sq_stage<TC, L>(area2, x, true, g);
    load_slice<L>(x, irow + ((scale ? d : half) - 1) * H);
    sq_pass<TC, L, false, false>(z, x, g.limb(area2, g.c, 0), 0u, 0u, x, nullptr, n, kc.npn, g);
    if (!scale) store_slice<L>(inv + (p * ent + d - 1) * H + g.t * L, z);
    copy_slice<L>(x, y);
    sq_pass<TC, L, false, false>(y, z, g.limb(area, g.c, 0), 0u, 0u, z, nullptr, n, kc.npn, g);
    load_slice<L>(z, left(p, d) + H + g.t * L);
    chain_reduce_once<TC, L>(y, 0u, n);
    chain_reduce_once<TC, L>(y, chain_add<TC, L>(y, y, z), n);
    load_slice<L>(z, right(p, d) + H + g.t * L);
    chain_reduce_once<TC, L>(y, chain_add<TC, L>(y, y, z), n);
  }
  uint32_t* e = table + ((size_t)(pos0 + p) * ent + d - 1) * S + g.t * L;
  store_slice<L>(e, x);
  store_slice<L>(e + H, y);
}

}  // namespace

// Time per product of one warp (us) when every scheduler holds `warps` warps of
// a layout, as measured on GB300 with encryption's passes of one row (Mul and
// MatMul, which also choose by it, run passes of two as well and hold other
// numbers of registers): few ciphertexts run fastest with many lanes a chain,
// many with few.  2048 bits, window 12: 608 ciphertexts take 0.31 ms
// with 16 lanes a chain (0.67 with 4), 4,864 take 0.99 ms with 4 (1.25 with 2
// or 16), 131,072 take 23.5 ms with 2, 23.9 with 4 and 30.9 with 16.
double sq_pass_cost(int H, int logtc, double warps) {
  static const double lat[3][5] = {{6.8, 3.9, 2.7, 0, 1.8}, {0, 13.2, 7.2, 4.4, 3.3}, {0, 29, 15.3, 8.1, 5.4}};
  static const double thr[3][5] = {{4.67, 2.35, 1.35, 0, 0.56}, {0, 9.3, 4.76, 2.71, 1.54}, {0, 20.6, 10.7, 5.5, 3.4}};
  const int r = H == 32 ? 0 : H == 64 ? 1 : 2;
  return std::max(lat[r][logtc], thr[r][logtc] * warps);
}

static int sm_count() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return std::max(sms, 1);
}

cudaError_t launch_sq_encrypt(int S, const KeyConst& kc, const EncArgs& a, uint32_t* out, size_t count, uint32_t* err,
                              cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  const int H = S / 2;
  const double scheds = 4.0 * sm_count();
  // Shares: several warps on each ciphertext, while the chain of products and
  // not the pipe sets the time: over the multiprocessors of a cluster up to two
  // warps a scheduler (more in one multiprocessor only slow each other down),
  // then in one block up to four.  One ciphertext (2048 bits, window 12) takes
  // 0.053 ms with 32 warps in 8 blocks, 0.059 with 16 in 4, 0.081 with 8 in one
  // and 0.306 with one; 76 take 0.073 ms with 16 and 0.081 with 8; of 3072
  // bits one takes 0.088, 0.103 and 0.173 ms with 32, 16 and 8.
  for (int blocks = 8; blocks > 2; blocks >>= 1) {
    if ((double)count * blocks * kClusterWarps > 2.0 * scheds) continue;
    HG_DISPATCH_SQ16(H, {
      Modulus<TC * L> m;
      std::copy(kc.hn, kc.hn + H, m.n);
      const cudaError_t e = blocks == 8 ? launch_cluster<TC, L, 8>(m, kc, a, out, count, err, st)
                                        : launch_cluster<TC, L, 4>(m, kc, a, out, count, err, st);
      if (e != cudaSuccess) return e;
    });
    count_launches(1);
    return cudaGetLastError();
  }
  for (int warps = kShareWarps; warps > 1; warps >>= 1) {
    if ((double)count * warps > 4.0 * scheds) continue;
    HG_DISPATCH_SQ16(H, {
      Modulus<TC * L> m;
      std::copy(kc.hn, kc.hn + H, m.n);
      const unsigned blocks = (unsigned)count;
      switch (warps) {
        case 8: k_sq_encrypt<TC, L, 8><<<blocks, 256, enc_smem<TC, L, 8>(), st>>>(m, kc, a, out, count, err); break;
        case 4: k_sq_encrypt<TC, L, 4><<<blocks, 128, enc_smem<TC, L, 4>(), st>>>(m, kc, a, out, count, err); break;
        default: k_sq_encrypt<TC, L, 2><<<blocks, 64, enc_smem<TC, L, 2>(), st>>>(m, kc, a, out, count, err); break;
      }
    });
    count_launches(1);
    return cudaGetLastError();
  }
  int best = -1;
  double best_cost = 1e300;
  for (int l = 0; l < 5; ++l) {
    if ((H != 32 && l == 0) || (H == 32 && l == 3)) continue;
    const size_t ipw = (size_t)16 >> l;
    const double per = std::ceil((double)((count + ipw - 1) / ipw) / scheds);
    const double cost = sq_pass_cost(H, l, per);
    if (cost < best_cost) {
      best_cost = cost;
      best = l;
    }
  }
  HG_DISPATCH_SQ(H, best, {
    Modulus<TC * L> m;
    std::copy(kc.hn, kc.hn + H, m.n);
    const size_t smem = enc_smem<TC, L, 1>();
    constexpr int IPW = SqLanes<TC, L>::IPW;
    k_sq_encrypt<TC, L, 1><<<(unsigned)((count + IPW - 1) / IPW), 32, smem, st>>>(m, kc, a, out, count, err);
  });
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_sq_bases(int S, const KeyConst& kc, const uint32_t* first, uint32_t* bases, cudaStream_t st) {
  HG_DISPATCH_SQ16(S / 2, k_sq_bases<TC, L><<<1, 64, 0, st>>>(kc, first, bases));
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_sq_level(int S, const KeyConst& kc, uint32_t* table, uint32_t* inv, const uint32_t* bases, int pos0,
                            size_t npos, int level, int subset, cudaStream_t st) {
  const size_t ent = (size_t)((1u << kc.w) - 1u);
  const bool scale = level == kc.w;
  const size_t lo = level < 0 || scale ? 1 : ((size_t)1 << level) + 1;
  const size_t hi = level < 0 ? 1 : scale ? ent : std::min(((size_t)1 << (level + 1)) - (subset ? 1 : 0), ent);
  if (hi < lo) return cudaSuccess;
  const size_t pairs = ((hi - lo + 1) * npos + 1) / 2;
  // 16 limbs a lane (12 at 3072 bits): enough groups for the small levels
  switch (S) {
    case 64: k_sq_level<2, 16><<<(unsigned)((pairs + 31) / 32), 128, 0, st>>>(kc, table, inv, bases, pos0, npos, level, subset); break;
    case 128: k_sq_level<4, 16><<<(unsigned)((pairs + 15) / 16), 128, 0, st>>>(kc, table, inv, bases, pos0, npos, level, subset); break;
    case 192: k_sq_level<8, 12><<<(unsigned)((pairs + 7) / 8), 128, 0, st>>>(kc, table, inv, bases, pos0, npos, level, subset); break;
    default: return cudaErrorInvalidValue;
  }
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace hg
