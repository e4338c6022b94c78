// Mul(ct, k) of ZPaillier keys by 64-bit scalars (sq_mul.cuh).  OU keys, whose
// modulus is no square, multiply with k_mul (paillier_kernels.cu).
#include <algorithm>
#include <atomic>
#include <cmath>

#include "sq_mul.cuh"

namespace hg {

namespace {

// Persistent, one warp per block; warps take groups of instances from the
// launch's counter.
//
// Bound: the fmaheavy pipe.  65,537 signed 64-bit scalars at 2048 bits took
// 22.0 ms as sliding windows of products modulo n^2 (84 of them at 8 H^2), with
// an inverse tree padded to 131,072 leaves; 16.2 ms here.
template <int TC, int L>
__global__ void __launch_bounds__(32) k_sq_mul(const __grid_constant__ KeyConst kc, const uint32_t* __restrict__ a,
                                               const int64_t* __restrict__ kk, uint32_t* __restrict__ out,
                                               size_t count, uint32_t* __restrict__ scratch, int wm, uint32_t* err,
                                               unsigned long long* ctr) {
  using G = SqLanes<TC, L>;
  __shared__ __align__(16) uint32_t area[2 * G::kDigit];
  const G g;
  uint32_t* tb = scratch + (size_t)blockIdx.x * mul_slots(wm) * 32 * L;
  uint32_t n[L];
  load_slice<L>(n, kc.n + g.t * L);
  const size_t groups = (count + G::IPW - 1) / G::IPW;
  for (size_t item = next_work(ctr, 1); item < groups; item = next_work(ctr, 1)) {
    const size_t inst = item * G::IPW + g.iw;
    const bool active = inst < count;
    sq_mul<TC, L>(n, kc, a, kk, out, active ? inst : count - 1, active, tb, wm, area, err, g);
  }
}

// Layouts by (limbs of n, log2 of the lanes per chain).
#define HG_DISPATCH_SQMUL(H, LOGTC, ...)                                        \
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

bool has_layout(int H, int logtc) {
  if (logtc < 1 || logtc > 4) return false;
  return H == 32 ? logtc != 3 : H == 64 ? true : logtc >= 2;
}

int resident_warps(int H, int logtc) {
  static std::atomic<int> cache[3][5];
  std::atomic<int>& slot = cache[H == 32 ? 0 : H == 64 ? 1 : 2][logtc];
  int v = slot.load(std::memory_order_relaxed);
  if (v == 0) {
    int dev = 0, sms = 0, per = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    [&]() -> cudaError_t {
      HG_DISPATCH_SQMUL(H, logtc, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_sq_mul<TC, L>, 32, 0));
      return cudaSuccess;
    }();
    v = sms * std::max(per, 1);
    slot.store(v, std::memory_order_relaxed);
  }
  return v;
}

}  // namespace

MulPlan mul_plan(int S, int wm, size_t count) {
  const int H = S / 2;
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const double scheds = 4.0 * std::max(sms, 1);
  MulPlan pl;
  double best = 1e300;
  for (int l = 1; l < 5; ++l) {
    if (!has_layout(H, l)) continue;
    const size_t ipw = (size_t)16 >> l;
    const size_t items = (count + ipw - 1) / ipw;
    const size_t cap = (size_t)resident_warps(H, l);
    const size_t rounds = (items + cap - 1) / cap;
    // The pass costs are the encryption's; Mul's own products of two rows take
    // (2, 32) at 2048 bits to 222 registers, two warps a scheduler.  A full round
    // of it is the fastest all the same (9,728 scalars 2.69 ms against 2.84 with
    // (4, 16), two rounds 4.87 against 4.98), but in a long column the four warps
    // of (4, 16) cover for each other: 32,768 9.10 against 8.21, 2^20 253 against
    // 233 (window 4).  1024 and 3072 bits keep their narrowest layout (2^17: 8.0 against
    // 8.7, 66.1 against 68.4).
    if (H == 64 && l == 1 && rounds > 2) continue;
    const size_t warps = (items + rounds - 1) / rounds;  // every warp the same number of items
    const double cost = (double)rounds * sq_pass_cost(H, l, std::ceil((double)warps / scheds));
    if (cost < best) {
      best = cost;
      pl.logtc = l;
      pl.warps = (int)warps;
    }
  }
  pl.scratch_words = (size_t)pl.warps * mul_slots(wm) * 32 * (size_t)(H >> pl.logtc);
  return pl;
}

// The most that any count's plan takes.
size_t mul_scratch_words(int S, int wm) {
  const int H = S / 2;
  size_t words = 0;
  for (int l = 1; l < 5; ++l)
    if (has_layout(H, l)) words = std::max(words, (size_t)resident_warps(H, l) * mul_slots(wm) * 32 * (size_t)(H >> l));
  return words;
}

cudaError_t launch_sq_mul(int S, const KeyConst& kc, const MulPlan& pl, const uint32_t* a, const int64_t* k,
                          uint32_t* out, size_t count, uint32_t* scratch, int wm, uint32_t* err,
                          unsigned long long* ctr, cudaStream_t st) {
  if (count == 0) return cudaSuccess;
  const cudaError_t e = cudaMemsetAsync(ctr, 0, sizeof(*ctr), st);
  if (e != cudaSuccess) return e;
  HG_DISPATCH_SQMUL(S / 2, pl.logtc,
                    k_sq_mul<TC, L><<<(unsigned)pl.warps, 32, 0, st>>>(kc, a, k, out, count, scratch, wm, err, ctr));
  count_launches(1);
  return cudaGetLastError();
}

}  // namespace hg
