// Persistent multi-key batch kernel: the templates, shared by the
// translation units that instantiate one layout variant set each
// (batch_v0.cu, batch_v1.cu, batch_v2.cu), so the variants compile in
// parallel.
//
// One launch runs a whole batch of jobs of different key sizes (1024, 2048,
// 3072 bits) and operations (encrypt, decrypt, add, scalar mul).  The host
// cuts every job into tiles of one warp pass (additions: four) and orders them
// by cost (most expensive first); each warp repeatedly takes the next tile from
// a device counter and runs the per-ciphertext body for the tile's key size:
// two digits modulo n (sq_encrypt.cuh, sq_mul.cuh) or a prime (sq_decrypt.cuh),
// additions modulo n^2 (paillier_ops.cuh).  All key sizes of one launch use the
// layouts of variant set V (tpi_for / tp_for): V = 0 and 1 are throughput
// layouts the autotuner picks from, V = 2 the latency layout (a whole warp per
// instance, a half warp per side of a decryption) that short requests run in.
#pragma once
#include <algorithm>

#include "batch.cuh"
#include "paillier_ops.cuh"
#include "sq_decrypt.cuh"
#include "sq_encrypt.cuh"
#include "sq_mul.cuh"

namespace hg {

namespace batch_detail {
constexpr int kBlock = 128;
constexpr int kWarps = kBlock / 32;
constexpr int kFirstClaimCycles = 4000;  // about 2 us
// Shared words of a warp: 80 a limb of a lane for the encryption's areas (up to
// 16, 32 and 6 limbs a lane), at least 48 a limb and 8 a limb of the prime for
// the decryption's.
template <int V>
constexpr int kAreaWords = V == 1 ? 80 * 32 : V == 0 ? 80 * 16 : 768;
}  // namespace batch_detail

template <int V, int S>
__device__ __noinline__ void run_tile(const BatchJob& job, const BatchTile& tile, uint32_t* ws, uint32_t* ysm,
                                         uint32_t* err) {
  constexpr int TPI = tpi_for(S, V), L = S / TPI;
  const int lane = threadIdx.x & 31;
  const size_t end = (size_t)tile.start + tile.count;
  if (job.op == kBatchDecrypt) {
    constexpr int SP = S / 2;
    // a group of TP lanes per side, TP / 2 a chain; both sides of a
    // ciphertext in neighbouring groups
    constexpr int TP = tp_for(SP, V), TC = TP / 2, LC = SP / TP, H = SP / 2;
    constexpr int UPW = 32 / (2 * TP);
    const SqLanes<TC, LC> g;
    const int side = g.iw & 1, unit_w = g.iw >> 1;
    uint32_t* zs = ysm + 2 * SqLanes<TC, LC>::kDigit;
    uint32_t* mm = zs + UPW * 2 * H;
    static_assert(2 * SqLanes<TC, LC>::kDigit + UPW * 2 * H + 4 * 2 * H <= batch_detail::kAreaWords<V>, "area");
    for (size_t wbase = tile.start; wbase < end; wbase += UPW) {
      const size_t inst = wbase + unit_w;
      const bool active = inst < end;
      __syncwarp();
      dec_pow_fixed<TC, LC>(job.kc, job.sc, side, (const uint32_t*)job.in0, active ? inst : end - 1, active, ws, ysm,
                            zs + g.iw * H, err, g);
      __syncwarp();
      // 8 lanes a ciphertext
#pragma unroll 1
      for (int u0 = 0; u0 < UPW; u0 += 4) {
        const int u = min(u0 + lane / 8, UPW - 1);
        const bool mine = u0 + lane / 8 < UPW && wbase + u < end;
        dec_tail<H / 8>(job.kc, job.sc, zs + u * 2 * H, mine ? wbase + u : end - 1, mine, mm + (lane / 8) * 2 * H,
                        (int64_t*)job.out, (uint8_t*)job.aux, nullptr, nullptr, Codec{});
        __syncwarp();
      }
    }
    return;
  }
  const Group<TPI> g;
  uint32_t N[L];
  load_slice<L>(N, job.kc.N + g.t * L);
  const int lane_inst = lane / TPI;
  constexpr int IPW = 32 / TPI;
  if (job.op == kBatchEncrypt && job.kc.two_digit) {
    const SqLanes<TPI / 2, L> sg;
    uint32_t n[L];
    load_slice<L>(n, job.kc.n + sg.t * L);
    const EncArgs a{EncMode::kEncrypt, (const int64_t*)job.in0, nullptr, nullptr, (const uint32_t*)job.in1, nullptr,
                    Codec{}};
    for (size_t wbase = tile.start; wbase < end; wbase += IPW) {
      const size_t inst = wbase + lane_inst;
      const bool active = inst < end;
      __syncwarp();
      sq_encrypt<TPI / 2, L, 1, 1>(n, job.kc, a, (uint32_t*)job.out, active ? inst : end - 1, active, ysm, nullptr, err,
                                sg);
    }
  } else if (job.op == kBatchEncrypt) {
    for (size_t wbase = tile.start; wbase < end; wbase += IPW) {
      const size_t inst = wbase + lane_inst;
      const bool active = inst < end;
      encrypt_one<TPI, L>(job.kc, EncMode::kEncrypt, (const int64_t*)job.in0, nullptr, nullptr,
                          (const uint32_t*)job.in1, nullptr, (uint32_t*)job.out, active ? inst : end - 1, active, N,
                          g, err);
    }
  } else if (job.op == kBatchAdd) {
    for (size_t wbase = tile.start; wbase < end; wbase += IPW) {
      const size_t inst = wbase + lane_inst;
      const bool active = inst < end;
      add_one<TPI, L>(job.kc, (const uint32_t*)job.in0, (const uint32_t*)job.in1, (uint32_t*)job.out,
                      active ? inst : end - 1, active, N, g, err);
    }
  } else if (job.op == kBatchMul && job.kc.two_digit) {
    const SqLanes<TPI / 2, L> sg;
    uint32_t n[L];
    load_slice<L>(n, job.kc.n + sg.t * L);
    for (size_t wbase = tile.start; wbase < end; wbase += IPW) {
      const size_t inst = wbase + lane_inst;
      const bool active = inst < end;
      __syncwarp();
      sq_mul<TPI / 2, L>(n, job.kc, (const uint32_t*)job.in0, (const int64_t*)job.in1, (uint32_t*)job.out,
                         active ? inst : end - 1, active, ws, job.wm, ysm, err, sg);
    }
  } else if (job.op == kBatchMul) {
    const int ntab = 1 << (job.wm - 1);
    uint32_t* tb = ws + (size_t)lane_inst * ntab * S + g.t * L;
    for (size_t wbase = tile.start; wbase < end; wbase += IPW) {
      const size_t inst = wbase + lane_inst;
      const bool active = inst < end;
      mul_one<TPI, L>(job.kc, (const uint32_t*)job.in0, (const int64_t*)job.in1, (uint32_t*)job.out,
                      active ? inst : end - 1, active, tb, job.wm, N, g, err);
    }
  }
}

// The next tile, which lane 0 claims by a predicate.  Claimed in a branch
// (`if (lane == 0) atomicAdd`) lane 0 stayed apart from the other lanes, and a
// tile's instructions were issued twice.
__device__ __forceinline__ uint32_t next_tile(uint32_t* counter) {
  uint32_t t;
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %2, 0;\n\tmov.u32 %0, 0;\n\t"
      "@p atom.global.add.u32 %0, [%1], 1;\n\t}"
      : "=r"(t)
      : "l"(counter), "r"(threadIdx.x & 31u)
      : "memory");
  return __shfl_sync(kFull, t, 0);
}

// Four blocks per SM in the layouts that fit them: the server splits an SM's
// blocks between its regular and its short batches.
template <int V>
__global__ void __launch_bounds__(batch_detail::kBlock, V == 1 ? 1 : 4) k_batch(const BatchJob* __restrict__ jobs,
                                                  const BatchTile* __restrict__ tiles, uint32_t ntiles,
                                                  uint32_t* __restrict__ counter, uint32_t* __restrict__ scratch,
                                                  size_t warp_words, uint32_t* err) {
  __shared__ __align__(16) uint32_t ysm[batch_detail::kWarps][batch_detail::kAreaWords<V>];
  const int wib = threadIdx.x >> 5;
  uint32_t* ws = scratch + ((size_t)blockIdx.x * batch_detail::kWarps + wib) * warp_words;
  // The first claims go round the chip, one warp a block: warp 1 waits 2 us, warp
  // 2 four and warp 3 six, while the launch's blocks arrive.  Without that the
  // multiprocessors whose blocks arrived first take the chains four to a
  // scheduler.  1,025 decryptions of 3072 bits alone: 10.1 ms with the wait, 27.3
  // without, 4,096 of 2048 bits 8.4 and 16.6, 600 additions of 2048 bits 0.076 and
  // 0.104, one addition 0.031 and 0.032; a mixed batch of 47,452 operations 24.0
  // and 28.3, and 19.2 and 18.9 with the next batch queued behind it.
  const long long started = clock64();
  while (clock64() - started < (long long)wib * batch_detail::kFirstClaimCycles) {
  }
  while (true) {
    const uint32_t t = next_tile(counter);
    if (t >= ntiles) break;
    const BatchTile tile = tiles[t];
    const BatchJob& job = jobs[tile.job];
    switch (job.S) {
      case 64: run_tile<V, 64>(job, tile, ws, ysm[wib], err); break;
      case 128: run_tile<V, 128>(job, tile, ws, ysm[wib], err); break;
      case 192: run_tile<V, 192>(job, tile, ws, ysm[wib], err); break;
      default: break;
    }
  }
}


template <typename K>
int batch_occupancy_blocks(K kernel) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, batch_detail::kBlock, 0);
  return sms * (per > 0 ? per : 1);
}

// Dynamic shared memory that caps `kernel` at `cap` resident blocks per SM.
template <typename K>
size_t batch_smem_cap_pad(K kernel, int cap) {
  int dev = 0, per_sm = 0, reserved = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
  cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev);
  cudaFuncAttributes fa{};
  cudaFuncGetAttributes(&fa, kernel);
  // cap blocks fit in per_sm, cap + 1 do not
  const size_t per_block = (size_t)((double)per_sm / ((double)cap + 0.5));
  const size_t used = fa.sharedSizeBytes + (size_t)reserved;
  const size_t pad = per_block > used ? per_block - used : 0;
  cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100);
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)pad);
  return pad;
}

void count_launches(uint64_t n);

// The three entry points of one variant set, defined by batch_v<V>.cu.
#define HG_BATCH_VARIANT_ENTRY_POINTS(V)                                                                      \
  void batch_carveout_v##V(int pct) {                                                                       \
    cudaFuncSetAttribute(k_batch<V>, cudaFuncAttributePreferredSharedMemoryCarveout, pct);                  \
  }                                                                                                         \
  int batch_resident_blocks_v##V() { return batch_occupancy_blocks(k_batch<V>); }                          \
  size_t batch_smem_cap_v##V(int blocks_per_sm) { return batch_smem_cap_pad(k_batch<V>, blocks_per_sm); } \
  cudaError_t launch_batch_v##V(const BatchJob* jobs, const BatchTile* tiles, uint32_t ntiles,              \
                                uint32_t* counter, uint32_t* scratch, size_t warp_words, uint32_t* err,     \
                                int grid, cudaStream_t st, size_t dyn_smem) {                               \
    k_batch<V><<<grid, batch_detail::kBlock, dyn_smem, st>>>(jobs, tiles, ntiles, counter, scratch,         \
                                                             warp_words, err);                              \
    count_launches(1);                                                                                      \
    return cudaGetLastError();                                                                              \
  }

}  // namespace hg
