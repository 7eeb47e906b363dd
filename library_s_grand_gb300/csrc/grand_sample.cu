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

__host__ __device__ inline void philox4x32_10(uint32_t (&c)[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const unsigned long long p0 = 0xD2511F53ull * c[0];
    const unsigned long long p1 = 0xCD9E8D57ull * c[2];
    const uint32_t hi0 = (uint32_t)(p0 >> 32), lo0 = (uint32_t)p0;
    const uint32_t hi1 = (uint32_t)(p1 >> 32), lo1 = (uint32_t)p1;
    const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
    c[0] = n0;
    c[1] = lo1;
    c[2] = n2;
    c[3] = lo0;
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

__device__ __forceinline__ uint32_t flip_threshold(float p) {
  // p * 2^32 is exact in FP32 (a power-of-two scale); truncate, clamp p >= 1
  const float s = p * 4294967296.0f;
  return s >= 4294967295.0f ? 0xFFFFFFFFu : (s <= 0.0f ? 0u : (uint32_t)s);
}

// One warp per shot, a block's warps in strides of the grid.  The positions' thresholds are
// formed once per block, in shared memory, a lane's four of a group side by side.  Flips
// are rare: a group is asked once whether it has any, and their columns then go straight
// into the lanes' syndrome (and logical) words, from which the entries are stored
// coalesced; an error record's entries are the lanes' own comparisons.
//
// Bound by the generator's products, 20 of 32 x 32 -> 64 bits per four positions (with a
// quarter of the other instructions taken out -- keys held in registers -- the time stayed
// the same).  65536 shots of the 720-mechanism DEM: 60 us, 128 when every word was scanned for
// flips and the thresholds formed per shot.
template <bool ERRORS>
__global__ void __launch_bounds__(256, 8) sample_kernel(DevCode cd, const float *p,
                                                     unsigned long long seed,
                                                     unsigned long long first_shot, int num_shots,
                                                     int *records) {
  extern __shared__ uint4 s_thr[];  // per group of 128 positions and lane: those of 32u + lane
  const int lane = threadIdx.x & 31;
  const int mpad = (cd.m + 127) & ~127;
  for (int j = threadIdx.x; j < mpad; j += blockDim.x)  // (zeros past the last position)
    reinterpret_cast<uint32_t *>(s_thr)[(j & ~127) + 4 * (j & 31) + ((j >> 5) & 3)] =
        j < cd.m ? flip_threshold(__ldg(p + j)) : 0u;
  __syncthreads();
  const uint32_t k0 = (uint32_t)seed, k1 = (uint32_t)(seed >> 32);
  const int nwarps = gridDim.x * 8;
  const bool dem = cd.family == kDem;
  const int nw = cd.nw, nlw = dem ? cd.nlw : 0;
#pragma unroll 1
  for (int i = blockIdx.x * 8 + (threadIdx.x >> 5); i < num_shots; i += nwarps) {
    const unsigned long long shot = first_shot + (unsigned long long)i;
    int *rec = records + (size_t)i * cd.rec_len;
    uint32_t s_lane = 0u, l_lane = 0u;  // syndrome / detector word `lane`, logical word `lane`
    // flips: 128 positions per group, four words of one block per lane
#pragma unroll 1
    for (int j0 = 0; j0 < mpad; j0 += 128) {
      uint32_t c[4] = {(uint32_t)(j0 / 4 + lane), (uint32_t)shot, (uint32_t)(shot >> 32),
                       0x47524E44u};
      philox4x32_10(c, k0, k1);
      const uint4 thr = s_thr[j0 / 4 + lane];
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
  int grid = (num_shots + 7) / 8;
  if (grid > sm_count * 8) grid = sm_count * 8;
  const size_t smem = sizeof(uint32_t) * ((cd.m + 127) & ~127);  // at most 16 KB
  if (cd.input_kind == kInErrors)
    sample_kernel<true><<<grid, 256, smem, s>>>(cd, d_p, seed, first_shot, num_shots, d_records);
  else
    sample_kernel<false><<<grid, 256, smem, s>>>(cd, d_p, seed, first_shot, num_shots, d_records);
  return cudaGetLastError();
}

}  // namespace grand
