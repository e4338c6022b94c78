// CRT decryption of a few ciphertexts: the exponentiation of decrypt_kernels.cu
// arranged for the shortest chain of dependent steps.
//
// The layouts there go through a factor's limbs one by one, a shuffle and two
// rows of multiply-adds each: 33 dependent steps a squaring at 2048 bits. Here
// one block does one side of one ciphertext and forms a product at once: its
// columns are spread over the block, every lane sums a quarter of the products
// of two columns.
//
// Limbs have 28 bits, so that a column's sum fits 64 bits: a product is one
// multiply-add without a carry, and instead of settling carries a limb takes
// what its three lower neighbours' columns hand up and may reach 2^28 + 2.
// Digits are X0 - X1 n as in sqmod.cuh, of E limbs, rho = 2^(28 E). With c_k =
// 2^(28 k) / rho mod n, n' = -1/n mod rho, and t_k the low E limbs of T, Th the
// high ones, reducing is one more such sum:
//   T0 = X0 Y0,                          Z0 = Th + sum t_k c_k
//   T1 = X0 Y1 + X1 Y0 + m,              Z1 = Th + sum t_k c_k
// where m = sum t_k (n' 2^(28 k) mod rho), t of T0, makes T0 + m n = Z0 rho:
// c_k rho = 2^(28 k) + (n' 2^(28 k) mod rho) n, whatever the limbs t_k. With n
// below 2^b (b = 32 H) a sum of E such terms is below 2^(b + 28) 1.01 E, so Z <
// 2^(b + 28) 1.05 E <= 2^(28 E - 4) and T < 2^(56 E): nothing is subtracted.
//
// Warps have a role: 0 X0 Y0 of operation t; 1, 2 and 3 X1 Y0, X0 Y1 and m of
// the operation before, since digit 0 never needs digit 1. Four barriers an
// operation: sums of T's columns, limbs of T, sums of Z's columns, limbs of Z.
//
// Bound by latency: shared-memory loads, ten dependent multiply-adds, shuffles
// and barriers, 1,620 cycles an operation at 2048 bits; the multiply-add pipe
// is a third busy. 8 decryptions of 2048 bits on GB300 took 1.01 ms against 1.71
// with 16 lanes a chain, of 3072 bits 2.25 against 4.88, of 1024 bits 0.41
// against 0.53. Limbs of 32 bits took 1.44 ms (three words a sum, carries settled
// by one warp), and every column all rows, zeros included, 1.28 ms.
#include <algorithm>

#include "sq_decrypt.cuh"

namespace hg {

namespace {

template <int H>
struct Lat {
  static constexpr int B = 28;
  static constexpr uint32_t M = (1u << B) - 1u;
  static constexpr int E = H == 16 ? 20 : H == 32 ? 38 : 57;
  static constexpr int NR = (E + 7) / 8 * 2, RP = 4 * NR;  // rows of a lane (even), of a number
  // NR rows meet a number in NR + E - 1 columns, E of them at most below rho
  static constexpr int NP = (NR + E) / 2;                  // pairs of columns of a quarter
  static constexpr int NPM = ((E + 1) / 2) + ((E - NR + 1) / 2) + ((E - 2 * NR + 1) / 2) + ((E - 3 * NR + 1) / 2);
  static constexpr int NW = (4 * NP + 31) / 32, NM = (NPM + 31) / 32;  // warps of a product, of m
  static constexpr int NF = (4 * E + 31) / 32;             // of a reduction: E columns, four lanes each
  static constexpr int kWarps = 3 * NW + NM;
  static constexpr int kShift = B * E - 32 * (H + 1);      // rho over sqmod.cuh's
  static constexpr int kOut = 32 * (H + 2) - B * E;        // bits up on the way out
  static constexpr int kPad = NR - 1;                      // odd: a lane's window of a number is 8-byte aligned
  static constexpr int kNum = 2 * NP + NR + 2;             // zeros, a number, zeros
  // 64-bit shared words: a role's four sums of each column, four columns of zeros below
  static constexpr int kCols = (4 + RP + E + 3) / 2 * 2, kPlane = 4 * kCols;
  static constexpr int kColsZ = (8 * NF + 15) / 16 * 16 + 4, kPlaneZ = 4 * kColsZ;
  static constexpr int kTw = (E + RP + 1) / 2 * 2;         // words of T
  static constexpr int kX0 = 2 * (4 * kPlane + 2 * kPlaneZ), kX1 = kX0 + 2 * kNum, kNp = kX1 + kNum,
                       kA0 = kNp + kNum, kT = kA0 + 2 * RP, kRaw = kT + 2 * kTw, kTab = kRaw + 2 * (H + 2);
  static_assert(kShift >= 0 && kShift <= B && kOut >= 0 && E > 3 * NR && kNum % 2 == 0 && kTab % 2 == 0, "limbs");
  static_assert(2 * NF <= kWarps && NW * 29 >= 2 * E && 2 * NP >= E + 1, "warps");
  static constexpr size_t smem(size_t slots, size_t steps) {
    return ((size_t)kTab + slots * 2 * RP) * 4 + (steps + 2) * 4;
  }
  // The most that any key takes: a program of w-bit windows has a squaring a bit
  // and a product for every w of them at most (build_prog).
  static constexpr size_t smem_bound() {
    size_t most = 0;
    for (size_t w = kMinDecWindow; w <= kMaxDecWindow; ++w) {
      const size_t ntab = (size_t)1 << (w - 1), b = smem(ntab + 1, ntab + 32 * H + 32 * H / w + 1);
      most = most > b ? most : b;
    }
    return most;
  }
};

// A quarter of columns k and k + 1 of a product: the NR rows at `a` by the NR + 1
// words at `b`, the first of which meets the last row in column k.
template <int NR>
__device__ __forceinline__ void lat_conv(uint64_t& s0, uint64_t& s1, const uint32_t* a, const uint32_t* b) {
  uint32_t x[NR], y[NR + 2];
#pragma unroll
  for (int u = 0; u < NR; u += 2) {
    const uint2 q = *reinterpret_cast<const uint2*>(a + u);
    x[u] = q.x;
    x[u + 1] = q.y;
  }
#pragma unroll
  for (int u = 0; u <= NR; u += 2) {
    const uint2 q = *reinterpret_cast<const uint2*>(b + u);
    y[u] = q.x;
    y[u + 1] = q.y;
  }
  uint64_t v0 = 0u, v1 = 0u;
  s0 = s1 = 0u;
#pragma unroll
  for (int u = 0; u < NR; u += 2) {
    s0 += (uint64_t)x[u] * y[NR - 1 - u];
    s1 += (uint64_t)x[u] * y[NR - u];
    v0 += (uint64_t)x[u + 1] * y[NR - 2 - u];
    v1 += (uint64_t)x[u + 1] * y[NR - 1 - u];
  }
  s0 += v0;
  s1 += v1;
}

// Sum of a column's four parts.
template <int W>
__device__ __forceinline__ uint64_t lat_col(const uint64_t* plane, int c) {
  return (plane[c] + plane[W + c]) + (plane[2 * W + c] + plane[3 * W + c]);
}

// Columns of neighbouring lanes -> limbs; the three lowest lanes only hand up.
template <int B>
__device__ __forceinline__ uint32_t lat_limb(uint64_t c) {
  constexpr uint32_t M = (1u << B) - 1u;
  const uint32_t r = ((uint32_t)c & M) + __shfl_up_sync(kFull, (uint32_t)(c >> B) & M, 1) +
                     __shfl_up_sync(kFull, (uint32_t)(c >> (2 * B)), 2);
  return (r & M) + __shfl_up_sync(kFull, r >> B, 1);
}

template <int H>
__global__ void __launch_bounds__(32 * Lat<H>::kWarps)
    k_dec_latency(const __grid_constant__ KeyConst kc, const __grid_constant__ SecConst sc,
                  const uint32_t* __restrict__ ct, uint32_t* __restrict__ z, uint32_t* err) {
  using A = Lat<H>;
  constexpr int E = A::E, RP = A::RP, NW = A::NW, NR = A::NR, B = A::B;
  constexpr int TC = H == 32 ? 16 : 8, L = H / TC;  // for the ways in and out
  extern __shared__ __align__(16) uint32_t lat_smem[];
  uint64_t* const planes = reinterpret_cast<uint64_t*>(lat_smem);  // by role, then a reduction's by chain
  uint32_t* const tab = lat_smem + A::kTab;                        // [slot][digit][RP]
  const int ntab = 1 << (sc.wd - 1);
  const int slots = ntab + 1;  // odd powers, the square
  // operation t: the factor's place in shared memory, 0: square
  int* const codes = reinterpret_cast<int*>(tab + slots * 2 * RP) + 1;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // roles in the order 0, 1, 3, 2, which spreads a square's over the schedulers
  const int role = warp < 2 * NW ? warp / NW : warp < 2 * NW + A::NM ? 3 : 2;
  const int w = warp - (role < 2 ? role * NW : role == 3 ? 2 * NW : 2 * NW + A::NM);
  const int chain = role ? 1 : 0, id = w * 32 + lane;
  const size_t i = blockIdx.x >> 1;
  const int side = blockIdx.x & 1;
  const uint32_t np = sc.np1[side];

  const uint16_t* prog = sc.prog[side];
  int len = sc.prog_len;
  while (len > 0 && prog[len - 1] == kOpNop) --len;  // the shorter program's padding
  // as in dec_pow_side: operation 0 squares into slot ntab, t < ntab makes slot
  // t, then the program
  const int last = ntab + len - 1, start = sc.start[side];
  for (int j = threadIdx.x; j < A::kTab + slots * 2 * RP; j += blockDim.x) lat_smem[j] = 0u;
  for (int j = (int)threadIdx.x - 1; j <= last + 1; j += blockDim.x) {
    int e = -1;
    if (j > 0 && j < ntab) e = ntab;
    if (j >= ntab && j <= last && prog[j - ntab] != kOpSquare) e = prog[j - ntab];
    codes[j] = e < 0 ? 0 : A::kTab + e * 2 * RP;
  }
  __syncthreads();
  uint32_t* const raw = lat_smem + A::kRaw;
  for (int j = threadIdx.x; j < E; j += blockDim.x) lat_smem[A::kNp + A::kPad + j] = sc.fold[side][E * E + j];
  uint32_t n[L];
  const SqLanes<TC, L> g;
  if (warp == 0) {
    const uint32_t* src = ct + i * (4 * H);
    if (side == 0) {
      // c < n^2 (decryptor.cc:21-23)
      const bool ok = raw_below<TC, 2 * L>(src, kc.N);
      if (!ok && lane == 0) atomicOr(err, kErrCtRange);
    }
    load_slice<L>(n, sc.P[side] + g.t * L);
    uint32_t x[L];
    sq_from_raw<TC, L, 4 * H>(x, src, n, np, g);
    if (g.iw == 0) {
#pragma unroll
      for (int j = 0; j < L; ++j) raw[g.c * (H + 2) + g.t * L + j] = x[j];
    }
  }
  // this lane's quarter of the rows and pair of columns in it
  int quarter = id / A::NP, pair = id % A::NP;
  if (role == 3) {
    quarter = 0;
    pair = id;
    while (quarter < 4 && pair >= (E - quarter * NR + 1) / 2) pair -= (E - quarter++ * NR + 1) / 2;
  }
  const bool has = quarter < 4;
  if (!has) quarter = pair = 0;
  const bool cut = role == 3 && NR * quarter + 2 * pair + 1 >= E;  // m ends below rho
  const int row = NR * quarter, a_tab = row + (role == 2 ? RP : 0);
  const int b_at = A::kPad + 2 * pair - (NR - 1) + (role == 3 ? A::kNp : role == 1 ? A::kX1 : A::kX0);
  const int b_step = role & 1 ? 0 : A::kNum;
  uint64_t* const plane = planes + role * A::kPlane + 4;  // the sums that this warp makes, or reads
  uint64_t* const put = plane + quarter * A::kCols + row + 2 * pair;
  // the column whose limb it makes
  const int own = 29 * w + lane - 3;
  const bool makes_t = role < 2 && 29 * w < 2 * E, makes_z = role < 2 && 29 * w < E;
  uint32_t* const T = lat_smem + A::kT + chain * A::kTw;
  uint64_t* const plane_z = planes + 4 * A::kPlane + chain * A::kPlaneZ + 4;
  // its part of a reduction, of chain fc, and the constants of that
  const int fc = warp >= A::NF ? 1 : 0, fid = (warp - fc * A::NF) * 32 + lane, fcol = fid >> 2, frow = NR * (lane & 3);
  const bool folds = warp < 2 * A::NF && fcol < E;
  uint32_t cr[NR];
#pragma unroll
  for (int u = 0; u < NR; ++u) cr[u] = (folds && frow + u < E) ? sc.fold[side][(frow + u) * E + fcol] : 0u;
  const uint32_t* const fold_t = lat_smem + A::kT + fc * A::kTw + frow;
  uint64_t* const put_z = planes + 4 * A::kPlane + fc * A::kPlaneZ + (lane & 3) * A::kColsZ + 4 + fcol;
  __syncthreads();
  if (role < 2 && id < E) {
    // limb id of the digit times 2^kShift
    const uint32_t* d = raw + chain * (H + 2);
    const int at = B * id - A::kShift, q = at >> 5;
    const uint32_t lo = q >= 0 ? d[q] : 0u, hi = q + 1 < H + 2 ? d[q + 1] : 0u;
    tab[chain * RP + id] = (q < H + 2 ? __funnelshift_r(lo, hi, at & 31) : 0u) & A::M;
    lat_smem[(chain ? A::kX1 : A::kX0) + A::kPad + id] = tab[chain * RP + id];
    if (!chain) lat_smem[A::kA0 + id] = tab[id];
  }
  __syncthreads();

  // digits 1 in the first turn and digits 0 in the last one make numbers that
  // nothing reads
  int next = codes[-chain];
#pragma unroll 1
  for (int turn = 0; turn <= last + 1; ++turn) {
    const int t = turn - chain, par = t & 1, code = next;
    next = codes[min(t + 1, last)];
    if (role != 2 || code) {
      const int a = role == 3 ? A::kT + row : code ? code + a_tab : A::kA0 + par * RP + row;
      uint64_t s0, s1;
      lat_conv<NR>(s0, s1, lat_smem + a, lat_smem + b_at + par * b_step);
      if (has) *reinterpret_cast<ulonglong2*>(put) = make_ulonglong2(s0, cut ? 0u : s1);
    }
    __syncthreads();
    if (makes_t) {
      uint64_t c = lat_col<A::kCols>(plane, own);
      if (chain) {
        const uint64_t m = lat_col<A::kCols>(plane + 2 * A::kPlane, own);
        c += (code ? lat_col<A::kCols>(plane + A::kPlane, own) : c) + m;
      }
      const uint32_t v = lat_limb<B>(c);
      if (lane >= 3 && own < 2 * E) T[own] = v;
    }
    __syncthreads();
    if (folds) {
      uint64_t v[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int u = 0; u < NR; u += 2) {
        const uint2 q = *reinterpret_cast<const uint2*>(fold_t + u);
        v[u & 2] += (uint64_t)q.x * cr[u];
        v[(u & 2) + 1] += (uint64_t)q.y * cr[u + 1];
      }
      *put_z = (v[0] + v[1]) + (v[2] + v[3]);
    }
    __syncthreads();
    if (makes_z) {
      uint32_t v = lat_limb<B>(lat_col<A::kColsZ>(plane_z, own) + (own >= 0 ? T[E + own] : 0u));
      if (lane >= 3 && own < E) {
        if (t < ntab) {
          if (t >= 0) tab[((t == 0 ? ntab : t) * 2 + chain) * RP + own] = v;
          const int from = t + 1 == ntab ? start : t <= 0 ? 0 : -1;
          if (from >= 0) v = tab[(from * 2 + chain) * RP + own];
        }
        lat_smem[(chain ? A::kX1 : A::kX0 + (par ^ 1) * A::kNum) + A::kPad + own] = v;
        if (!chain) lat_smem[A::kA0 + (par ^ 1) * RP + own] = v;
      }
    }
    __syncthreads();
  }

  // both digits as words, 2^kOut times; then H + 2 limbs off them
  if (threadIdx.x < 2) {
    const uint32_t* x = lat_smem + (threadIdx.x ? A::kX1 : A::kX0 + ((last + 1) & 1) * A::kNum) + A::kPad;
    uint32_t* d = raw + threadIdx.x * (H + 2);
    uint64_t acc = 0u;
    int have = A::kOut, at = 0;
#pragma unroll 1
    for (int j = 0; j < E; ++j) {
      acc += (uint64_t)x[j] << have;  // x[j] may reach 2^28
      have += B;
      if (have >= 32) {
        d[at++] = (uint32_t)acc;
        acc >>= 32;
        have -= 32;
      }
    }
  }
  __syncthreads();
  if (warp == 0) {
    const uint32_t* src = raw + g.c * (H + 2);
    uint32_t V[L], O[L], x[L], ov = 0u, c1 = 0u;
#pragma unroll
    for (int j = 0; j < L; ++j) {
      V[j] = src[g.t * L + j];
      O[j] = 0u;
    }
    const bool top = g.t == TC - 1;
#pragma unroll 1
    for (int j = H; j < 2 * H + 2; j += 2) {
      // the words above the number are zeros
      const uint32_t lo = top && j == H ? src[H] : 0u, hi = top && j == H ? src[H + 1] : 0u;
      sq_redc_step<TC, L>(V, O, ov, c1, n, np, lo, g);
      sq_redc_step<TC, L>(O, V, ov, c1, n, np, hi, g);
    }
    sq_settle<TC, L>(x, V, O, c1, n, g);
    dec_check<TC, L>(x, sc, side, g);
    if (g.iw == 0 && g.c == 1) store_slice<L>(z + (2 * i + side) * H + g.t * L, x);
  }
}

#define HG_DISPATCH_LAT(H_, ...)                           \
  switch (H_) {                                            \
    case 16: { constexpr int H = 16; __VA_ARGS__; } break; \
    case 32: { constexpr int H = 32; __VA_ARGS__; } break; \
    case 48: { constexpr int H = 48; __VA_ARGS__; } break; \
    default: return cudaErrorInvalidValue;                 \
  }

}  // namespace

int dec_latency_limbs(int H) { return H == 16 ? Lat<16>::E : H == 32 ? Lat<32>::E : Lat<48>::E; }

cudaError_t launch_dec_latency(int H_, const KeyConst& kc, const SecConst& sc, const uint32_t* ct, size_t count,
                               uint32_t* z, uint32_t* err, cudaStream_t st) {
  const size_t ntab = (size_t)1 << (sc.wd - 1), steps = ntab + (size_t)sc.prog_len;
  HG_DISPATCH_LAT(H_, {
    const size_t smem = Lat<H>::smem(ntab + 1, steps);
    constexpr size_t kBound = Lat<H>::smem_bound();
    static_assert(kBound <= 227 * 1024, "shared memory");
    if (smem > kBound) return cudaErrorInvalidValue;
    if (smem > 48 * 1024) {
      // The limit is the function's, for all threads and keys: every call sets it to
      // the same bound, so that none takes another's away before its launch.
      const cudaError_t e = cudaFuncSetAttribute(k_dec_latency<H>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBound);
      if (e != cudaSuccess) return e;
    }
    k_dec_latency<H><<<(unsigned)(2 * count), 32 * Lat<H>::kWarps, smem, st>>>(kc, sc, ct, z, err);
  });
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace hg
