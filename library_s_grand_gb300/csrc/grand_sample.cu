// grand_sample.cu -- on-device shot generation for registered codes (sm_103a).
//
// No upstream counterpart: upstream draws its shots in Python (numpy / stim,
// Create_Files/*) and ships them to the decoder as int32 rows.  Here a kernel
// draws i.i.d. flips of every error position (CSS: qubit, DEM: mechanism) with
// per-position probabilities, forms the syndrome / detectors and true logical
// flips, and writes the code's int32 records straight into device memory for
// grand_engine_decode_device: a statistical run never moves shots over PCIe or
// C2C.
//
// Random numbers: Philox4x32-10 (Salmon, Moraes, Dror, Shaw, "Parallel random
// numbers: as easy as 1, 2, 3", SC 2011), a counter-based generator: output
// block = Philox(counter, key) with no state, so every (seed, shot, position)
// has its own fixed draw whatever the launch shape.  Key = the 64-bit seed;
// counter = {group, shot low, shot high, 0x47524E44}; lane l of a warp computes
// block (32g + l) and uses word u for position 128g + 32u + l.  A position
// flips when its 32-bit word is below floor(p * 2^32) (p = 1: 2^32 - 1).
#include <cuda_runtime.h>

#include "grand_device.cuh"
#include "grand_host.h"

namespace grand {

constexpr uint32_t kPhiloxM0 = 0xD2511F53u, kPhiloxM1 = 0xCD9E8D57u;
constexpr uint32_t kPhiloxW0 = 0x9E3779B9u, kPhiloxW1 = 0xBB67AE85u;
constexpr uint32_t kPhiloxTag = 0x47524E44u;

__device__ __forceinline__ void mul_wide(uint32_t a, uint32_t b, uint32_t &hi, uint32_t &lo) {
  const unsigned long long p = (unsigned long long)a * b;
  hi = (uint32_t)(p >> 32);
  lo = (uint32_t)p;
}

// The first two rounds multiply words that depend on the block alone (its number, then that
// product's words) or on the shot alone, never on both: each half is formed once.
struct PhiloxBlock {
  uint32_t x0, x1, x2;  // after two rounds: word 0 and word 2 less the shot's part, word 1
};
struct PhiloxShot {
  uint32_t x0, x2, x3;  // the shot's part of words 0 and 2, word 3
};
__device__ __forceinline__ PhiloxBlock philox_block(uint32_t block, uint32_t k1) {
  PhiloxBlock r;
  uint32_t hi;
  mul_wide(kPhiloxM0, block, hi, r.x2);
  mul_wide(kPhiloxM1, hi ^ kPhiloxTag ^ k1, r.x0, r.x1);
  return r;
}
__device__ __forceinline__ PhiloxShot philox_shot(unsigned long long shot, uint32_t k0, uint32_t k1) {
  PhiloxShot r;
  uint32_t hi, lo;
  mul_wide(kPhiloxM1, (uint32_t)(shot >> 32), hi, lo);
  r.x0 = lo ^ (k0 + kPhiloxW0);
  mul_wide(kPhiloxM0, hi ^ (uint32_t)shot ^ k0, hi, r.x3);
  r.x2 = hi ^ (k1 + kPhiloxW1);
  return r;
}
// The other eight rounds.
__device__ __forceinline__ void philox_finish(const PhiloxBlock &b, const PhiloxShot &s,
                                              const uint32_t (&keys)[16], uint32_t (&c)[4]) {
  c[0] = b.x0 ^ s.x0;
  c[1] = b.x1;
  c[2] = b.x2 ^ s.x2;
  c[3] = s.x3;
#pragma unroll
  for (int r = 2; r < 10; ++r) {
    uint32_t hi0, lo0, hi1, lo1;
    mul_wide(kPhiloxM0, c[0], hi0, lo0);
    mul_wide(kPhiloxM1, c[2], hi1, lo1);
    c[0] = hi1 ^ c[1] ^ keys[2 * r - 4];
    c[1] = lo1;
    c[2] = hi0 ^ c[3] ^ keys[2 * r - 3];
    c[3] = lo0;
  }
}

__device__ __forceinline__ uint32_t flip_threshold(float p) {
  // p * 2^32 is exact in FP32 (a power-of-two scale); truncate, clamp p >= 1
  const float s = p * 4294967296.0f;
  return s >= 4294967295.0f ? 0xFFFFFFFFu : (s <= 0.0f ? 0u : (uint32_t)s);
}

// One block per SM, its warps drawing the block's shots one at a time (a shared counter: in
// fixed strides the warps that the scheduler prefers ended early, and the rest ran at 42 of
// 64 warps).  The positions' thresholds and the blocks' halves of the first two rounds are
// formed once per block, in shared memory, the thresholds of a lane's four positions side by
// side.  Flips are rare: a group is asked once whether it has any, and their columns then
// go straight into the lanes' syndrome (and logical) words, from which the entries are stored
// coalesced; an error record's entries are the lanes' own comparisons.
//
// Bound by issue: the products (16 of 32 x 32 -> 64 bits per four positions) keep their pipe
// 51 % busy, logic and comparisons theirs 59 %.  65536 shots of the 720-mechanism DEM: 50 us
// (60 with all 20 products, 64 warps per SM in strides and keys formed in every group;
// 2 x 1024, 3 x 512 or 2 x 768 threads per SM are 4 to 16 us slower, 1 x 512 as well).
constexpr int kSampleThreads = 1024;

template <bool ERRORS>
__global__ void __launch_bounds__(kSampleThreads, 1) sample_kernel(DevCode cd, const float *p,
                                                                   unsigned long long seed,
                                                                   unsigned long long first_shot, int num_shots,
                                                                   int *records) {
  __shared__ unsigned s_next;  // (goes on past the last shot, which can be the largest int)
  extern __shared__ uint4 s_thr[];  // per group of 128 positions and lane: those of 32u + lane
  const int lane = threadIdx.x & 31;
  const int mpad = (cd.m + 127) & ~127;
  for (int j = threadIdx.x; j < mpad; j += blockDim.x)  // (zeros past the last position)
    reinterpret_cast<uint32_t *>(s_thr)[(j & ~127) + 4 * (j & 31) + ((j >> 5) & 3)] =
        j < cd.m ? flip_threshold(__ldg(p + j)) : 0u;
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  uint32_t *s_blk = reinterpret_cast<uint32_t *>(s_thr + mpad / 4);  // the blocks' halves, by word
  const int nblk = mpad / 4;
  for (int j = threadIdx.x; j < nblk; j += blockDim.x) {
    const PhiloxBlock h = philox_block((uint32_t)j, k1);
    s_blk[j] = h.x0;
    s_blk[nblk + j] = h.x1;
    s_blk[2 * nblk + j] = h.x2;
  }
  uint32_t keys[16];  // of rounds 3 .. 10 (held: formed anew they were a fifth of the instructions)
#pragma unroll
  for (int r = 2; r < 10; ++r) {
    keys[2 * r - 4] = k0 + (uint32_t)r * kPhiloxW0;
    keys[2 * r - 3] = k1 + (uint32_t)r * kPhiloxW1;
    asm volatile("" : "+r"(keys[2 * r - 4]), "+r"(keys[2 * r - 3]));
  }
  // the block's shots, drawn by its warps
  const unsigned last = (unsigned)((long long)num_shots * (blockIdx.x + 1) / gridDim.x);
  if (threadIdx.x == 0) s_next = (unsigned)((long long)num_shots * blockIdx.x / gridDim.x);
  __syncthreads();
  const bool dem = cd.family == kDem;
  const int nw = cd.nw, nlw = dem ? cd.nlw : 0;
#pragma unroll 1
  for (;;) {
    unsigned i = 0;
    if (lane == 0) i = atomicAdd(&s_next, 1u);
    i = __shfl_sync(kFull, i, 0);
    if (i >= last) break;
    const unsigned long long shot = first_shot + i;
    int *rec = records + (size_t)i * cd.rec_len;
    const PhiloxShot half = philox_shot(shot, k0, k1);
    uint32_t s_lane = 0u, l_lane = 0u;  // syndrome / detector word `lane`, logical word `lane`
    // flips: 128 positions per group, four words of one block per lane
#pragma unroll 1
    for (int j0 = 0; j0 < mpad; j0 += 128) {
      const int blk = j0 / 4 + lane;
      uint32_t c[4];
      philox_finish(PhiloxBlock{s_blk[blk], s_blk[nblk + blk], s_blk[2 * nblk + blk]}, half, keys, c);
      const uint4 thr = s_thr[blk];
      const bool f[4] = {c[0] < thr.x, c[1] < thr.y, c[2] < thr.z, c[3] < thr.w};
      if constexpr (ERRORS) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (j0 + 32 * u + lane < cd.m) rec[j0 + 32 * u + lane] = f[u] ? 1 : 0;
      } else if (__any_sync(kFull, f[0] || f[1] || f[2] || f[3])) {
#pragma unroll 1
        for (int u = 0; u < 4; ++u) {
          const bool mine = u == 0 ? f[0] : (u == 1 ? f[1] : (u == 2 ? f[2] : f[3]));
#pragma unroll 1
          for (uint32_t bits = __ballot_sync(kFull, mine); bits; bits &= bits - 1u) {
            // XOR of the flipped columns, and of their rows of L
            const int col = j0 + 32 * u + __ffs((int)bits) - 1;
            if (lane < nw) s_lane ^= __ldg(cd.cols + (size_t)col * cd.nwp + lane);
            if (lane < nlw) l_lane ^= __ldg(cd.lcols + (size_t)col * cd.nlw + lane);
          }
        }
      }
    }
    if constexpr (!ERRORS) {
#pragma unroll 1
      for (int r = lane; r - lane < cd.R; r += 32) {
        const uint32_t word = __shfl_sync(kFull, s_lane, r >> 5);
        if (r < cd.R) rec[r] = (int)((word >> lane) & 1u);
      }
#pragma unroll 1
      for (int j = lane; dem && j - lane < cd.n_logicos; j += 32) {
        const uint32_t word = __shfl_sync(kFull, l_lane, j >> 5);
        if (j < cd.n_logicos) rec[cd.R + j] = (int)((word >> lane) & 1u);
      }
    }
  }
}

cudaError_t launch_sample(const DevCode &cd, const float *d_p, unsigned long long seed,
                          unsigned long long first_shot, int num_shots, int *d_records,
                          int sm_count, cudaStream_t s) {
  if (num_shots <= 0) return cudaSuccess;
  int grid = num_shots;
  if (grid > sm_count) grid = sm_count;
  const int mpad = (cd.m + 127) & ~127;
  const size_t smem = sizeof(uint32_t) * (mpad + 3 * (mpad / 4));  // at most 28 KB
  if (cd.input_kind == kInErrors)
    sample_kernel<true><<<grid, kSampleThreads, smem, s>>>(cd, d_p, seed, first_shot, num_shots, d_records);
  else
    sample_kernel<false><<<grid, kSampleThreads, smem, s>>>(cd, d_p, seed, first_shot, num_shots, d_records);
  return cudaGetLastError();
}

}  // namespace grand
