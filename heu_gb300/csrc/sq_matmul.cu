// heu.numpy MatMul of a ciphertext matrix by an integer plaintext matrix
// (numpy/evaluator.cc:208-292) for ZPaillier keys, in two digits (sqmod.cuh):
// out(i,j) = prod_k x(i,k)^y(k,j) mod n^2.
//
// Like matmul_kernels.cu, every row gets tables of the subset products of
// chunks of b bases, and every output is a Horner pass over the bit planes of
// its exponents.  Entries are kept as in sq_encrypt.cuh, as an integer Y0 and
// y with Y = Y0 (1 - y n): a lookup then multiplies by an integer of n's length
// (4 H^2 multiply-adds instead of 8 H^2) and adds y; a plane's squaring doubles
// the sum.  For that the bases' digits are divided: y = X1 / X0 mod n, by one
// batch inversion modulo n of all X0 of a block of rows (a product tree; three
// products of H limbs a base).  A base that shares a factor with n (no
// ciphertext) leaves the call to the kernels modulo n^2.
//
// Bound: the fmaheavy pipe.  256 x 128 @ 128 x 32 with 16-bit plaintexts at 2048
// bits took 16.3 ms modulo n^2 (8 bases a chunk) and takes 10.1 ms here (6).
#include <algorithm>
#include <cmath>

#include "sq_encrypt.cuh"

namespace hg {

namespace {

// Where base k of row i goes: unit (row, chunk) and entry of the unit.
struct Place {
  size_t unit;
  size_t entry;
};
__device__ __forceinline__ Place place_of(size_t i, int k, int nch, int b) {
  const int c = k / b;
  return {i * (size_t)nch + c, ((size_t)1 << (k - c * b)) - 1};
}

// Bases into the form: digits of C rho, digit 0 to the table entry and to the
// tree's leaves, digit 1 to the entry's second half.  Bases past K are 1.
template <int TC, int L>
__global__ void __launch_bounds__(128) k_mm_bases(const __grid_constant__ KeyConst kc, const uint32_t* __restrict__ x,
                                                  size_t r0, size_t rows, int K, int b, int nch,
                                                  uint32_t* __restrict__ T, uint32_t* __restrict__ leaves,
                                                  uint32_t* err) {
  using G = SqLanes<TC, L>;
  constexpr int H = G::H, S = 2 * H;
  __shared__ __align__(16) uint32_t areas[4][2 * G::kDigit];
  const G g;
  uint32_t* area = areas[threadIdx.x >> 5];
  const size_t Kp = (size_t)nch * b, total = rows * Kp, ent = ((size_t)1 << b) - 1;
  const size_t first = ((size_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * G::IPW;
  if (first >= total) return;
  const bool active = first + g.iw < total;
  const size_t u = active ? first + g.iw : total - 1;
  const size_t i = u / Kp;
  const int k = (int)(u % Kp);
  const uint32_t* src = x + ((r0 + i) * (size_t)K + min(k, K - 1)) * S;
  const bool ok = raw_below<TC, L>(src, kc.N);
  if (active && !ok && k < K && g.lane == g.base) atomicOr(err, kErrCtRange);
  uint32_t n[L], z[L], w[L];
  load_slice<L>(n, kc.n + g.t * L);
  sq_from_raw<TC, L, S>(z, src, n, kc.npn, g);
  // times the constant's integer; its second factor joins y later
  load_slice<L>(w, kc.rz + g.t * L);
  sq_stage<TC, L>(area, w, false, g);
  sq_pass<TC, L, false>(z, z, g.limb(area, 0, 0), 0u, 0u, z, nullptr, n, kc.npn, g);
  if (k >= K) load_slice<L>(z, kc.one + g.c * H + g.t * L);
  const Place p = place_of(i, k, nch, b);
  if (!active) return;
  store_slice<L>(T + (p.unit * ent + p.entry) * S + g.c * H + g.t * L, z);
  if (g.c == 0) store_slice<L>(leaves + u * H + g.t * L, z);
}

// y = X1 / X0 of every base (the leaves now hold rho^2 / X0), and the inverses
// to the tables' side; a group does two bases, one per chain.
template <int TC, int L>
__global__ void __launch_bounds__(128) k_mm_log(const __grid_constant__ KeyConst kc, size_t rows, int K, int b,
                                                int nch, uint32_t* __restrict__ T, const uint32_t* __restrict__ leaves,
                                                uint32_t* __restrict__ inv) {
  using G = SqLanes<TC, L>;
  constexpr int H = G::H, S = 2 * H;
  __shared__ __align__(16) uint32_t areas[4][2 * G::kDigit];
  const G g;
  uint32_t* area = areas[threadIdx.x >> 5];
  const size_t Kp = (size_t)nch * b, total = rows * Kp, ent = ((size_t)1 << b) - 1;
  const size_t first = ((size_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * 2 * G::IPW;
  if (first >= total) return;
  const size_t u = min(first + 2 * g.iw + g.c, total - 1);
  const size_t i = u / Kp;
  const int k = (int)(u % Kp);
  const Place p = place_of(i, k, nch, b);
  uint32_t n[L], x[L], y[L];
  load_slice<L>(n, kc.n + g.t * L);
  uint32_t* e = T + (p.unit * ent + p.entry) * S + H + g.t * L;
  load_slice<L>(x, e);
  sq_stage<TC, L>(area, x, true, g);
  load_slice<L>(x, leaves + u * H + g.t * L);
  store_slice<L>(inv + (p.unit * ent + p.entry) * H + g.t * L, x);
  sq_pass<TC, L, false, false>(y, x, g.limb(area, g.c, 0), 0u, 0u, x, nullptr, n, kc.npn, g);
  chain_reduce_once<TC, L>(y, 0u, n);
  load_slice<L>(x, kc.rz + H + g.t * L);
  if (k >= K) {
#pragma unroll
    for (int j = 0; j < L; ++j) x[j] = 0u;
  }
  chain_reduce_once<TC, L>(y, chain_add<TC, L>(y, y, x), n);
  // one lane group may hold the last base twice
  if (first + 2 * g.iw + g.c < total) store_slice<L>(e, y);
}

// Product tree modulo n over H-limb nodes, two nodes a group (one per chain):
// node = a b / rho; on the way down u = rho^2 / node gives rho^2 / a = u b / rho.
template <int TC, int L>
__global__ void __launch_bounds__(128) k_half_up(const __grid_constant__ KeyConst kc,
                                                 const uint32_t* __restrict__ lower, size_t lower_count,
                                                 uint32_t* __restrict__ upper) {
  using G = SqLanes<TC, L>;
  constexpr int H = G::H;
  __shared__ __align__(16) uint32_t areas[4][2 * G::kDigit];
  const G g;
  uint32_t* area = areas[threadIdx.x >> 5];
  const size_t total = (lower_count + 1) / 2;
  const size_t first = ((size_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * 2 * G::IPW;
  if (first >= total) return;
  const size_t q = min(first + 2 * g.iw + g.c, total - 1);
  const bool pair = 2 * q + 1 < lower_count;
  uint32_t n[L], a[L], z[L];
  load_slice<L>(n, kc.n + g.t * L);
  load_slice<L>(a, lower + (2 * q + (pair ? 1 : 0)) * H + g.t * L);
  sq_stage<TC, L>(area, a, true, g);
  load_slice<L>(a, lower + 2 * q * H + g.t * L);
  sq_pass<TC, L, false, false>(z, a, g.limb(area, g.c, 0), 0u, 0u, a, nullptr, n, kc.npn, g);
  select_slice<L>(z, pair, z, a);
  store_slice<L>(upper + q * H + g.t * L, z);
}

template <int TC, int L>
__global__ void __launch_bounds__(128) k_half_down(const __grid_constant__ KeyConst kc, uint32_t* __restrict__ lower,
                                                   size_t lower_count, const uint32_t* __restrict__ upper) {
  using G = SqLanes<TC, L>;
  constexpr int H = G::H;
  __shared__ __align__(16) uint32_t areas[4][2 * G::kDigit];
  const G g;
  uint32_t* area = areas[threadIdx.x >> 5];
  const size_t total = (lower_count + 1) / 2;
  const size_t first = ((size_t)blockIdx.x * 4 + (threadIdx.x >> 5)) * 2 * G::IPW;
  if (first >= total) return;
  const bool mine = first + 2 * g.iw + g.c < total;
  const size_t q = mine ? first + 2 * g.iw + g.c : total - 1;
  const bool pair = 2 * q + 1 < lower_count;
  uint32_t n[L], u[L], a[L], z[L];
  load_slice<L>(n, kc.n + g.t * L);
  load_slice<L>(u, upper + q * H + g.t * L);
#pragma unroll 1
  for (int s = 0; s < 2; ++s) {
    // s = 0: the first child's, by the second; s = 1 the other way round
    load_slice<L>(a, lower + (2 * q + (s == 0 && pair ? 1 : 0)) * H + g.t * L);
    sq_stage<TC, L>(area, a, true, g);
    if (s == 0) {
      sq_pass<TC, L, false, false>(z, u, g.limb(area, g.c, 0), 0u, 0u, u, nullptr, n, kc.npn, g);
      select_slice<L>(z, pair, z, u);
    } else {
      sq_pass<TC, L, false, false>(a, u, g.limb(area, g.c, 0), 0u, 0u, u, nullptr, n, kc.npn, g);
    }
  }
  if (!mine) return;
  store_slice<L>(lower + 2 * q * H + g.t * L, z);
  if (pair) store_slice<L>(lower + (2 * q + 1) * H + g.t * L, a);
}

// out(r0 + i, j): Horner over the planes, lookups by masks
// masks[(j * P + plane) * nch + c] = bits of y'(bc .. bc + b - 1, j) in `plane`.
// One warp per block.
template <int TC, int L>
__global__ void __launch_bounds__(32) k_mm_planes(const __grid_constant__ KeyConst kc, const uint32_t* __restrict__ T,
                                                  const uint8_t* __restrict__ masks, size_t r0, size_t rows,
                                                  int Ncols, int P, int nch, int b, int plane_run,
                                                  uint32_t* __restrict__ out) {
  using G = SqLanes<TC, L>;
  constexpr int H = G::H, S = 2 * H, kDigit = G::kDigit, V = G::kVec;
  // two entries in flight, the sum of the y, the squaring's digit 0
  __shared__ __align__(16) uint32_t area[6 * kDigit];
  const G g;
  const size_t total = rows * (size_t)Ncols;
  const size_t first = (size_t)blockIdx.x * G::IPW;
  const bool active = first + g.iw < total;
  const size_t u = active ? first + g.iw : total - 1;
  const size_t i = u / Ncols;
  const int j = (int)(u % Ncols);
  const size_t ent = ((size_t)1 << b) - 1;
  const uint32_t* tab = T + i * nch * ent * S;
  const uint8_t* mk = masks + (size_t)j * P * nch;
  const int last = P * nch;  // then the output's radix
  // lookup e is chunk e % nch of plane P - 1 - e / nch
  int fc = 0, fp = P - 1;  // chunk and plane of the next fetch
  auto fetch = [&](int e, int buf) {
    const uint32_t* src;
    if (e >= last) {
      src = kc.e0;
    } else {
      const uint32_t m = mk[(size_t)fp * nch + fc];
      src = m ? tab + ((size_t)fc * ent + m - 1) * S : kc.e1;
      if (++fc == nch) {
        fc = 0;
        --fp;
      }
    }
    src += g.c * H + g.t * L;
    uint32_t* dst = g.limb(area + buf * 2 * kDigit, g.c, 0);
#pragma unroll
    for (int v = 0; v < L / V; ++v) cp_async(dst + g.slice_at(v), src + v * V, V * 4);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  uint32_t* sum = g.limb(area + 4 * kDigit, 0, 0);
  uint32_t* sq = g.limb(area + 5 * kDigit, 0, 0);
  uint32_t n[L], x[L], carry = 0u, top = 0u;
  load_slice<L>(n, kc.n + g.t * L);
  // the sum's limbs settled, its top word in `top`
  auto settle_sum = [&](uint32_t(&w)[L]) {
    sq_get<TC, L>(w, sum, g);
    top += chain_settle<TC, L>(w, carry);
    carry = 0u;
  };
  fetch(0, 0);
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  __syncwarp();
  {
    uint32_t s[L];
    sq_get<TC, L>(s, g.limb(area, g.c, 0), g);
    if (g.c == 1) sq_put<TC, L>(sum, s, g);
#pragma unroll
    for (int q = 0; q < L; ++q) x[q] = g.c ? 0u : s[q];
  }
  fetch(1, 1);
  int chunk = 1 % nch, run = 0;  // chunk of lookup e
#pragma unroll 1
  for (int e = 1, buf = 1; e <= last; ++e, buf ^= 1) {
    if (chunk == 0 && e < last) {
      // next plane: square the digits, double the sum
      uint32_t w[L];
      settle_sum(w);
      const uint32_t twice = chain_add<TC, L>(w, w, w);
      top = 2u * top + twice;
      __syncwarp();
      if (g.c == 1) sq_put<TC, L>(sum, w, g);
      if (g.c == 0) sq_put<TC, L>(sq, x, g);
      __syncwarp();
      sq_pass<TC, L, false>(x, x, sq, (uint32_t)g.c, 0u, x, nullptr, n, kc.npn, g);
      if (++run == plane_run) {
        // back below n: sum * rho^2 / rho^2 would be two products; rho^2 / rho
        // once and 1 / rho once more are the same two
        run = 0;
#pragma unroll 1
        for (int s = 0; s < 2; ++s) {
          uint32_t f[L];
          if (s == 0) {
            load_slice<L>(f, kc.rho2 + g.t * L);
          } else {
#pragma unroll
            for (int q = 0; q < L; ++q) f[q] = g.t == 0 && q == 0 ? 1u : 0u;
          }
          __syncwarp();
          sq_pass<TC, L, false, false>(w, f, sum, 0u, g.c ? top : 0u, f, nullptr, n, kc.npn, g);
          top = 0u;
          __syncwarp();
          if (g.c == 1) sq_put<TC, L>(sum, w, g);
        }
      }
    }
    if (++chunk >= nch) chunk = 0;
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncwarp();
    if (e < last) fetch(e + 1, buf ^ 1);
    uint32_t* cur = area + buf * 2 * kDigit;
    if (g.c == 1) {
      uint32_t s[L], y[L];
      sq_get<TC, L>(s, sum, g);
      sq_get<TC, L>(y, g.limb(cur, 1, 0), g);
      s[0] = add_cc(s[0], y[0]);
#pragma unroll
      for (int q = 1; q < L; ++q) s[q] = addc_cc(s[q], y[q]);
      carry = addc(carry, 0u);
      sq_put<TC, L>(sum, s, g);
    }
    __syncwarp();
    sq_pass<TC, L, false>(x, x, g.limb(cur, 0, 0), 0u, 0u, x, nullptr, n, kc.npn, g);
  }
  // X1 += X0 * sum
  uint32_t w[L], p0[L];
  settle_sum(w);
  __syncwarp();
  if (g.c == 1) sq_put<TC, L>(sum, w, g);
#pragma unroll
  for (int q = 0; q < L; ++q) p0[q] = __shfl_sync(kFull, x[q], g.c ? g.lane - TC : g.lane);
  __syncwarp();
  sq_pass<TC, L, false, false>(w, p0, sum, 0u, g.c ? top : 0u, p0, nullptr, n, kc.npn, g);
  chain_reduce_once<TC, L>(w, 0u, n);
  const uint32_t over = chain_add<TC, L>(w, x, w);
  chain_reduce_once<TC, L>(w, over, n);
  select_slice<L>(x, g.c == 1, w, x);
  uint32_t r[L];
  sq_to_raw<TC, L>(r, x, area, n, kc.npn, g);
  if (active) store_slice<L>(out + ((r0 + i) * (size_t)Ncols + j) * S + g.c * H + g.t * L, r);
}

// 16 limbs a lane (12 at 3072 bits) for the preparation.
#define HG_DISPATCH_MM(H, ...)                                                  \
  switch (H) {                                                                  \
    case 32: { constexpr int TC = 2, L = 16; __VA_ARGS__; } break;              \
    case 64: { constexpr int TC = 4, L = 16; __VA_ARGS__; } break;              \
    case 96: { constexpr int TC = 8, L = 12; __VA_ARGS__; } break;              \
    default: return cudaErrorInvalidValue;                                      \
  }
// The widest layouts, for a tree's small levels.
#define HG_DISPATCH_MM16(H, ...)                                                \
  switch (H) {                                                                  \
    case 32: { constexpr int TC = 16, L = 2; __VA_ARGS__; } break;              \
    case 64: { constexpr int TC = 16, L = 4; __VA_ARGS__; } break;              \
    case 96: { constexpr int TC = 16, L = 6; __VA_ARGS__; } break;              \
    default: return cudaErrorInvalidValue;                                      \
  }
// Layouts of the planes, by (limbs of n, log2 of the lanes per chain).
#define HG_DISPATCH_PLANES(H, LOGTC, ...)                                       \
  switch ((H) * 8 + (LOGTC)) {                                                  \
    case 257: { constexpr int TC = 2, L = 16; __VA_ARGS__; } break;             \
    case 258: { constexpr int TC = 4, L = 8; __VA_ARGS__; } break;              \
    case 260: { constexpr int TC = 16, L = 2; __VA_ARGS__; } break;             \
    case 513: { constexpr int TC = 2, L = 32; __VA_ARGS__; } break;             \
    case 514: { constexpr int TC = 4, L = 16; __VA_ARGS__; } break;             \
    case 515: { constexpr int TC = 8, L = 8; __VA_ARGS__; } break;              \
    case 516: { constexpr int TC = 16, L = 4; __VA_ARGS__; } break;             \
    case 770: { constexpr int TC = 4, L = 24; __VA_ARGS__; } break;             \
    case 771: { constexpr int TC = 8, L = 12; __VA_ARGS__; } break;             \
    case 772: { constexpr int TC = 16, L = 6; __VA_ARGS__; } break;             \
    default: return cudaErrorInvalidValue;                                      \
  }

// Nodes of a level up to which the widest layout is as fast: its warps take two
// products each, 8 per SM.
size_t wide_nodes() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return (size_t)16 * std::max(sms, 1);
}

template <int TC, int L>
unsigned pair_blocks(size_t count) {
  const size_t per = 4 * 2 * (size_t)SqLanes<TC, L>::IPW;
  return (unsigned)((count + per - 1) / per);
}

}  // namespace

// Chunk width with the fewest passes per row: tables of 2^b - 1 - b entries at
// two passes each, and N P lookups per chunk at one.
int sq_matmul_chunk(size_t K, size_t N, size_t P) {
  int best = 1;
  double cost = 1e300;
  for (int b = 1; b <= 8; ++b) {
    const double nch = std::ceil((double)K / b);
    const double c = nch * (2.0 * ((1 << b) - 1 - b) + 3.5 * b + (double)N * (double)P);
    if (c < cost) {
      cost = c;
      best = b;
    }
  }
  return best;
}

cudaError_t launch_mm_bases(int S, const KeyConst& kc, const uint32_t* x, size_t r0, size_t rows, int K, int b,
                            uint32_t* T, uint32_t* leaves, uint32_t* err, cudaStream_t st) {
  const int nch = (K + b - 1) / b;
  const size_t total = rows * (size_t)nch * b;
  HG_DISPATCH_MM(S / 2, {
    const size_t per = 4 * (size_t)SqLanes<TC, L>::IPW;
    k_mm_bases<TC, L><<<(unsigned)((total + per - 1) / per), 128, 0, st>>>(kc, x, r0, rows, K, b, nch, T, leaves, err);
  });
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_mm_log(int S, const KeyConst& kc, size_t rows, int K, int b, uint32_t* T, const uint32_t* leaves,
                          uint32_t* inv, cudaStream_t st) {
  const int nch = (K + b - 1) / b;
  HG_DISPATCH_MM(S / 2, k_mm_log<TC, L><<<pair_blocks<TC, L>(rows * (size_t)nch * b), 128, 0, st>>>(
                            kc, rows, K, b, nch, T, leaves, inv));
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_half_up(int S, const KeyConst& kc, const uint32_t* lower, size_t lower_count, uint32_t* upper,
                           cudaStream_t st) {
  const size_t total = (lower_count + 1) / 2;
  if (total <= wide_nodes()) {
    HG_DISPATCH_MM16(S / 2,
                     k_half_up<TC, L><<<pair_blocks<TC, L>(total), 128, 0, st>>>(kc, lower, lower_count, upper));
  } else {
    HG_DISPATCH_MM(S / 2,
                   k_half_up<TC, L><<<pair_blocks<TC, L>(total), 128, 0, st>>>(kc, lower, lower_count, upper));
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_half_down(int S, const KeyConst& kc, uint32_t* lower, size_t lower_count, const uint32_t* upper,
                             cudaStream_t st) {
  const size_t total = (lower_count + 1) / 2;
  if (total <= wide_nodes()) {
    HG_DISPATCH_MM16(S / 2,
                     k_half_down<TC, L><<<pair_blocks<TC, L>(total), 128, 0, st>>>(kc, lower, lower_count, upper));
  } else {
    HG_DISPATCH_MM(S / 2,
                   k_half_down<TC, L><<<pair_blocks<TC, L>(total), 128, 0, st>>>(kc, lower, lower_count, upper));
  }
  count_launches(1);
  return cudaGetLastError();
}

cudaError_t launch_mm_planes(int S, const KeyConst& kc, const uint32_t* T, const uint8_t* masks, size_t r0,
                             size_t rows, int Ncols, int P, int K, int b, uint32_t* out, cudaStream_t st) {
  const int H = S / 2, nch = (K + b - 1) / b;
  // planes until the doubled sum could pass its 32-bit top word
  int run = 28;
  while (run > 1 && ((size_t)(nch + 2) << run) >= ((size_t)1 << 30)) --run;
  const size_t total = rows * (size_t)Ncols;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  int best = -1;
  double best_cost = 1e300;
  for (int l = 1; l < 5; ++l) {
    if ((H == 32 && l == 3) || (H == 96 && l == 1)) continue;
    const size_t ipw = (size_t)16 >> l;
    const double per = std::ceil((double)((total + ipw - 1) / ipw) / (4.0 * std::max(sms, 1)));
    const double cost = sq_pass_cost(H, l, per);
    if (cost < best_cost) {
      best_cost = cost;
      best = l;
    }
  }
  HG_DISPATCH_PLANES(H, best, {
    constexpr int IPW = SqLanes<TC, L>::IPW;
    k_mm_planes<TC, L><<<(unsigned)((total + IPW - 1) / IPW), 32, 0, st>>>(kc, T, masks, r0, rows, Ncols, P, nch, b,
                                                                          run, out);
  });
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace hg
