// CRT decryption (decryptor.cc:32-53) in two kernels:
//   k_dec_pow   c^(p-1) mod p^2 and c^(q-1) mod q^2 by sliding windows, in two
//               digits to the base of the prime (sqmod.cuh): the result's
//               second digit is, up to constants of the key, L_p(c^(p-1));
//   k_dec_tail  m_p, m_q, their CRT combination, the sign fold and decoding.
//
// Bound: the fmaheavy pipe (wide multiply-adds).  A squaring of the exponent's
// 1,024 at 2048 bits costs 4 H^2 multiply-adds with H = 32 limbs, against
// 8 H^2 of a Montgomery product modulo p^2, and a chain of a prime's limbs in
// one lane needs no shuffles but one and reads the prime from the constant
// bank.  65,536 decryptions on GB300: 206 ms with 64-bit rows modulo p^2, 160 ms
// with the columns of mont.cuh, 87 ms in two digits (84% of the issue bound of
// the products it makes).
#include <algorithm>
#include <atomic>
#include <cmath>

#include "sq_decrypt.cuh"

namespace hg {

void count_launches(uint64_t n);

namespace {

// Both primes by value: with one lane per chain the multiply-adds take them
// as constant-bank operands.
template <int H>
struct DecPrimes {
  uint32_t n[2][H];
};

// One side of a warp's instances: digit 1 of c^(p-1) mod p^2, to
// z[(2 i + side) H ..].  The exponent program and its table (2^(wd-1) odd
// powers, then the square) are as in build_prog.
template <int TC, int L, class Mod>
__device__ __forceinline__ void dec_pow_side(const Mod& n, const KeyConst& kc, const SecConst& sc, int side,
                                             const uint32_t* __restrict__ ct, size_t i, bool active, uint32_t* tb,
                                             uint32_t* area, uint32_t* __restrict__ z, uint32_t* err,
                                             const SqLanes<TC, L>& g) {
  constexpr int H = TC * L;
  const uint32_t np = sc.np1[side];
  const uint16_t* prog = sc.prog[side];
  const int ntab = 1 << (sc.wd - 1);
  const uint32_t* src = ct + i * (4 * H);
  if (side == 0) {
    // c < n^2 (decryptor.cc:21-23)
    const bool ok = raw_below<TC, 2 * L>(src, kc.N);
    if (active && !ok && g.lane == g.base) atomicOr(err, kErrCtRange);
  }
  uint32_t x[L];
  sq_from_raw<TC, L, 4 * H>(x, src, n, np, g);
  table_store<L>(tb, 0, g.lane, x);
  // one loop over the table's products and the program, so that each kind of
  // pass is compiled once: step 0 squares into slot ntab, step s < ntab makes
  // slot s from slot s - 1 and the square, the rest is the program
  const int steps = ntab + sc.prog_len;
#pragma unroll 1
  for (int s = 0; s < steps; ++s) {
    int e = -1;  // -1: square, else multiply by slot e
    if (s < ntab) {
      if (s > 0) e = ntab;
    } else {
      const uint16_t op = prog[s - ntab];
      if (op == kOpNop) break;  // only pads the shorter program
      if (op != kOpSquare) e = op;
    }
    if (s == 1) table_load<L>(x, tb, 0, g.lane);
    if (s == ntab) table_load<L>(x, tb, sc.start[side], g.lane);
    sq_stage<TC, L>(area, x, e >= 0, g);
    if (e < 0) {
      sq_pass<TC, L, false>(x, x, g.limb(area, 0, 0), (uint32_t)g.c, 0u, x, nullptr, n, np, g);
    } else {
      uint32_t y0[L];
      table_load<L>(x, tb, e, g.lane);
      table_load<L>(y0, tb, e, g.lane - g.c * TC);
      sq_pass<TC, L, true>(x, x, g.limb(area, 0, 0), 0u, 0u, y0, g.limb(area, 1, 0), n, np, g);
    }
    if (s < ntab) table_store<L>(tb, s == 0 ? ntab : s, g.lane, x);
  }
  dec_digit<TC, L>(x, sc, side, n, np, g);
  if (active && g.c == 1) store_slice<L>(z + (2 * i + side) * H + g.t * L, x);
}

// Resident warps per SM that the compiler must fit, one warp per block.  With 32
// limbs a lane 9 to 12 are the same three warps a scheduler: 168 registers, 396
// bytes of spills.  8 take 234 registers and none: 2^20 decryptions of 2048 bits
// 1,328 ms against 1,267 at 12, 65,536 88.1 against 86.8, but 14,592 (one round
// of 12) 20.3 against 21.0 and 29,184 38.5 against 42.9.
constexpr int dec_min_blocks(int L) { return L == 48 ? 8 : L == 32 ? 10 : L == 24 ? 12 : L == 16 ? 16 : L == 12 ? 18 : 20; }

// One warp per block: warps take (side, group of instances) items from the
// launch's counter, all first sides before the second ones.
template <int TC, int L>
__global__ void __launch_bounds__(32, dec_min_blocks(L))
    k_dec_pow(const __grid_constant__ DecPrimes<TC * L> primes, const __grid_constant__ KeyConst kc,
              const __grid_constant__ SecConst sc, const uint32_t* __restrict__ ct, size_t count,
              uint32_t* __restrict__ scratch, uint32_t* __restrict__ z, uint32_t* err, unsigned long long* ctr) {
  using G = SqLanes<TC, L>;
  __shared__ __align__(16) uint32_t area[2 * G::kDigit];
  const G g;
  const size_t slots = ((size_t)1 << (sc.wd - 1)) + 1;
  uint32_t* tb = scratch + (size_t)blockIdx.x * slots * 32 * L;
  const size_t groups = (count + G::IPW - 1) / G::IPW;
  for (size_t item = next_work(ctr, 1); item < 2 * groups; item = next_work(ctr, 1)) {
    const int side = item < groups ? 0 : 1;
    const size_t inst = (item - (side ? groups : 0)) * G::IPW + g.iw;
    const bool active = inst < count;
    const size_t i = active ? inst : count - 1;
    if constexpr (TC == 1) {
      if (side == 0)
        dec_pow_side<TC, L>(primes.n[0], kc, sc, 0, ct, i, active, tb, area, z, err, g);
      else
        dec_pow_side<TC, L>(primes.n[1], kc, sc, 1, ct, i, active, tb, area, z, err, g);
    } else {
      uint32_t n[L];
      load_slice<L>(n, sc.P[side] + g.t * L);
      dec_pow_side<TC, L>(n, kc, sc, side, ct, i, active, tb, area, z, err, g);
    }
  }
}

// dec_tail over all ciphertexts of a chunk; under 1% of the decryption.
template <int LT>
__global__ void __launch_bounds__(128) k_dec_tail(const __grid_constant__ KeyConst kc,
                                                  const __grid_constant__ SecConst sc,
                                                  const uint32_t* __restrict__ z, size_t count,
                                                  int64_t* __restrict__ out_i64, uint8_t* __restrict__ out_ovf,
                                                  uint32_t* __restrict__ out_mag, uint8_t* __restrict__ out_neg,
                                                  const __grid_constant__ Codec cd, size_t first) {
  constexpr int H = 8 * LT;
  __shared__ __align__(16) uint32_t mm[16][2 * H];
  const size_t inst = ((size_t)blockIdx.x * 128 + threadIdx.x) / 8;
  const bool active = inst < count;
  const size_t u = active ? inst : count - 1;
  dec_tail<LT>(kc, sc, z + u * 2 * H, first + u, active, mm[threadIdx.x / 8], out_i64, out_ovf, out_mag, out_neg, cd);
}

// Layouts by (limbs of a prime, log2 of the lanes per chain).
#define HG_DISPATCH_DEC(H, LOGTC, ...)                                          \
  switch ((H) * 8 + (LOGTC)) {                                                  \
    case 128: { constexpr int TC = 1, L = 16; __VA_ARGS__; } break;             \
    case 129: { constexpr int TC = 2, L = 8; __VA_ARGS__; } break;              \
    case 130: { constexpr int TC = 4, L = 4; __VA_ARGS__; } break;              \
    case 131: { constexpr int TC = 8, L = 2; __VA_ARGS__; } break;              \
    case 256: { constexpr int TC = 1, L = 32; __VA_ARGS__; } break;             \
    case 257: { constexpr int TC = 2, L = 16; __VA_ARGS__; } break;             \
    case 258: { constexpr int TC = 4, L = 8; __VA_ARGS__; } break;              \
    case 259: { constexpr int TC = 8, L = 4; __VA_ARGS__; } break;              \
    case 260: { constexpr int TC = 16, L = 2; __VA_ARGS__; } break;             \
    case 384: { constexpr int TC = 1, L = 48; __VA_ARGS__; } break;             \
    case 385: { constexpr int TC = 2, L = 24; __VA_ARGS__; } break;             \
    case 386: { constexpr int TC = 4, L = 12; __VA_ARGS__; } break;             \
    case 387: { constexpr int TC = 8, L = 6; __VA_ARGS__; } break;              \
    default: return cudaErrorInvalidValue;                                      \
  }

int layouts(int H) { return H == 32 ? 5 : 4; }

// Resident warps of the whole device in a layout, cached per device-wide kernel.
int resident_warps(int H, int logtc) {
  static std::atomic<int> cache[3][5];
  std::atomic<int>& slot = cache[H == 16 ? 0 : H == 32 ? 1 : 2][logtc];
  int v = slot.load(std::memory_order_relaxed);
  if (v == 0) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    [&]() -> cudaError_t {
      HG_DISPATCH_DEC(H, logtc, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_dec_pow<TC, L>, 32, 0));
      return cudaSuccess;
    }();
    v = sms * std::max(per, 1);
    slot.store(v, std::memory_order_relaxed);
  }
  return v;
}

// Time of one item (ms) when every scheduler holds `warps` warps of a layout,
// as measured on GB300 with the default windows: more lanes per chain shorten
// the chain of dependent steps but spend more shuffles per limb, so few
// ciphertexts run fastest in the widest layout and many in the narrowest.
// 2048 bits: 8 ciphertexts take 1.97 ms with 16 lanes a chain against 10.7 ms
// with one, 2,432 take 4.1 ms with 4 lanes (5.2 with 8, 6.0 with 2), 131,072
// take 169 ms with one lane against 180 with two.
double item_cost(int H, int logtc, double warps) {
  static const double lat[3][5] = {{1.32, 0.95, 0.78, 0.62, 0}, {10.2, 5.7, 2.9, 2.14, 1.96}, {29, 17.5, 8.6, 5.2, 0}};
  static const double thr[3][5] = {{0.85, 0.53, 0.31, 0.2, 0}, {6.5, 3.4, 1.98, 1.27, 0.83}, {20.3, 11.1, 5.95, 3.4, 0}};
  const int r = H == 16 ? 0 : H == 32 ? 1 : 2;
  return std::max(lat[r][logtc], thr[r][logtc] * warps);
}

// Digits between the two kernels, at most: every pair of launches ends with a
// part-filled chip. 2^20 ciphertexts of 2048 bits take 1,268 ms, and 1,336 in
// chunks of 32 MiB.
constexpr size_t kHandoffBytes = (size_t)128 << 20;

}  // namespace

DecryptPlan decrypt_plan(int Sp, const SecConst& sc, size_t count) {
  const int H = Sp / 2;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const double scheds = 4.0 * std::max(sms, 1);
  DecryptPlan pl;
  pl.chunk = std::min(count, kHandoffBytes / ((size_t)2 * H * 4));
  double best = 1e300;
  for (int l = 0; l < layouts(H); ++l) {
    const size_t ipw = (size_t)16 >> l;
    const size_t items = 2 * ((pl.chunk + ipw - 1) / ipw);
    const size_t cap = (size_t)resident_warps(H, l);
    const size_t rounds = (items + cap - 1) / cap;
    const size_t warps = (items + rounds - 1) / rounds;  // every warp the same number of items
    const double per = std::ceil((double)warps / scheds);
    const double cost = (double)rounds * item_cost(H, l, per);
    if (cost < best) {
      best = cost;
      pl.logtc = l;
      pl.warps = (int)warps;
    }
  }
  // up to two blocks a multiprocessor for decrypt_latency.cu: 2048 bits 1.01 ms
  // to 76 ciphertexts and 1.41 ms for 152, where the layouts above take 1.71 and
  // 1.72; 304 take 2.76 ms against 1.73.  3072 bits: 2.25 and 4.47 ms against
  // 4.90; 1024 bits: 0.41 against 0.53 ms, but 0.60 for 300.
  pl.latency = count <= (size_t)std::max(sms, 1);
  const size_t slots = ((size_t)1 << (sc.wd - 1)) + 1;
  pl.table_words = pl.latency ? 0 : (size_t)pl.warps * slots * 32 * (size_t)(H >> pl.logtc);
  pl.handoff_words = pl.chunk * 2 * (size_t)H;
  return pl;
}

// The most that any count's plan takes.
size_t decrypt_scratch_words(int Sp, const SecConst& sc) {
  const int H = Sp / 2;
  const size_t slots = ((size_t)1 << (sc.wd - 1)) + 1;
  size_t tables = 0;
  for (int l = 0; l < layouts(H); ++l)
    tables = std::max(tables, (size_t)resident_warps(H, l) * slots * 32 * (size_t)(H >> l));
  return tables + kHandoffBytes / 4;
}

cudaError_t launch_decrypt(int Sp, const KeyConst& kc, const SecConst& sc, const uint32_t* primes,
                           const DecryptPlan& pl, const uint32_t* ct, size_t count, int64_t* out_i64,
                           uint8_t* out_ovf, uint32_t* out_mag, uint8_t* out_neg, uint32_t* scratch, uint32_t* err,
                           unsigned long long* ctr, cudaStream_t st, const Codec& cd) {
  const int H = Sp / 2;
  uint32_t* z = scratch + pl.table_words;
  for (size_t off = 0; off < count; off += pl.chunk) {
    const size_t n = std::min(pl.chunk, count - off);
    cudaError_t e = cudaSuccess;
    if (pl.latency) {
      if ((e = launch_dec_latency(H, kc, sc, ct + off * 4 * H, n, z, err, st)) != cudaSuccess) return e;
    } else {
      if ((e = cudaMemsetAsync(ctr, 0, sizeof(*ctr), st)) != cudaSuccess) return e;
      HG_DISPATCH_DEC(H, pl.logtc, {
        DecPrimes<TC * L> pr;
        std::copy(primes, primes + 2 * TC * L, &pr.n[0][0]);
        const size_t items = 2 * ((n + SqLanes<TC, L>::IPW - 1) / SqLanes<TC, L>::IPW);
        k_dec_pow<TC, L><<<(unsigned)std::min(items, (size_t)pl.warps), 32, 0, st>>>(pr, kc, sc, ct + off * 4 * H, n,
                                                                                    scratch, z, err, ctr);
      });
      count_launches(1);
      if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    const unsigned blocks = (unsigned)((n + 15) / 16);
    switch (H) {
      case 16: k_dec_tail<2><<<blocks, 128, 0, st>>>(kc, sc, z, n, out_i64, out_ovf, out_mag, out_neg, cd, off); break;
      case 32: k_dec_tail<4><<<blocks, 128, 0, st>>>(kc, sc, z, n, out_i64, out_ovf, out_mag, out_neg, cd, off); break;
      case 48: k_dec_tail<6><<<blocks, 128, 0, st>>>(kc, sc, z, n, out_i64, out_ovf, out_mag, out_neg, cd, off); break;
      default: return cudaErrorInvalidValue;
    }
    count_launches(1);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

size_t decrypt_wave(int Sp) { return (size_t)resident_warps(Sp / 2, 0) * 16 / 2; }

}  // namespace hg
