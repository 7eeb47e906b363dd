// grand_front.cuh -- the chunk kernel (sm_103a): the shots of a batch whose codes have a guided
// search, from their records to their results.
//
// Each warp classifies one chunk (grand_chunk.cuh).  The block's open shots then make one
// list, drawn by its warps four at a time for the guided search (grand_guided.cuh), or
// fewer when that leaves warps without any: a chunk's open shots would otherwise
// follow one another on its own warp, and the batch wait for the unluckiest.  Last, each
// warp writes its chunk's results.  Blocks are scheduled by the hardware; no block waits
// for another.
//
// It is a kernel of its own, not a step of the persistent decode kernel, for its working
// set: there (46 KB of shared memory per block, 128 registers, 650 KB of code) the same
// search ran at 16 warps per SM out of 28 KB of L1 and missed the instruction caches
// (headline batch 80 us, 100000-shot mix 178 us, noisy [[288]] 164 us, where a kernel of its
// own took 48, 125 and 92 us with the same warp-per-shot search).
#pragma once

#include "grand_chunk.cuh"
#include "grand_guided.cuh"

namespace grand {

// A load whose value nothing uses, for the line it brings into L1.
__device__ __forceinline__ void touch_line(const void *p) {
#ifdef GRAND_HOST_EMULATION
  (void)p;
#else
  unsigned x;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(x) : "l"(p));
#endif
}
constexpr int kWarmTam = 192;  // active sets whose candidate counts are fetched ahead

struct ChunkArea {
  GuidedArea guided;
  FastArea fast;
};

template <bool MLK>
__global__ void __launch_bounds__(kChunkWarps * 32, kChunkMinBlocks) chunk_kernel(const DevBatch b) {
  __shared__ ChunkArea areas[kChunkWarps];
  __shared__ HotCode hot[kHotCodes];
  __shared__ uint16_t open[kChunkWarps * kMaxChunk];
  __shared__ int open_count, open_next, stats[3];
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int chunk = (int)blockIdx.x * kChunkWarps + wib;
  const bool has = (long long)chunk * b.chunk < (long long)b.num_shots;
  const unsigned tag = *reinterpret_cast<volatile unsigned *>(b.epoch) + 1u;
  const unsigned long long t_enter = b.profile ? global_ns() : 0ull;
  FastArea &F = areas[wib].fast;
  GuidedArea &A = areas[wib].guided;
  ChunkStats st{0, 0, 0};

  // the codes, and one load per 128-byte line of their tables and of the candidate counts
  // of small sets: the first blocks of an SM find its L1 empty, and this way the lines come
  // together, in place of one miss after another along the search's chains (one shot of
  // [[144]], waited for: 48.5 us, 51 without; batches of 1, 8 and 16 DEMs of 62 KB, of which
  // every block touches the first eight's: within 0.5 us of the time without)
  {
    const int n = b.num_codes < kHotCodes ? b.num_codes : kHotCodes;
    constexpr int kWords = (int)(sizeof(HotCode) / 8);
#pragma unroll 1
    for (int i = threadIdx.x; i < n * kWords; i += kChunkWarps * 32) {
      const int k = i / kWords;
      reinterpret_cast<unsigned long long *>(hot + k)[i - k * kWords] =
          __ldg(reinterpret_cast<const unsigned long long *>(static_cast<const HotCode *>(b.codes + k)) + i -
                k * kWords);
    }
    if (threadIdx.x == 0) open_count = open_next = stats[0] = stats[1] = stats[2] = 0;
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < n; ++k) {
      const int lines = hot[k].g_gs ? (hot[k].g_words + 31) >> 5 : 0;
#pragma unroll 1
      for (int i = threadIdx.x; i < lines; i += kChunkWarps * 32) touch_line(hot[k].g_rows + 32 * i);
    }
#pragma unroll 1
    for (int i = threadIdx.x; i < kWarmTam / 2; i += kChunkWarps * 32) touch_line(b.upto + 16 * i);
  }

  unsigned mine = 0u;
  if (has) {
    static_assert(4 * kLogBallots <= sizeof(A.item), "the logicals' ballots fit the items");
    mine = classify_chunk<MLK>(b, hot, chunk, b.chunk, F, reinterpret_cast<uint32_t *>(A.item), st);
  }
  if (mine) {
    int base = 0;
    if (lane == 0) base = atomicAdd(&open_count, __popc(mine));
    base = __shfl_sync(kFull, base, 0);
    if ((mine >> lane) & 1u)
      open[base + __popc(mine & ((1u << lane) - 1u))] = (uint16_t)((wib << 8) | lane);
  }
  __syncthreads();

  const int count = open_count;
  constexpr int kGroups = 32 / kGuidedLanes;
  int take = (count + kChunkWarps - 1) / kChunkWarps;
  if (take > kGroups) take = kGroups;
#pragma unroll 1
  while (count) {
    int at = 0;
    if (lane == 0) at = atomicAdd(&open_next, take);
    at = __shfl_sync(kFull, at, 0);
    if (at >= count) break;
    const int cnt = count - at < take ? count - at : take;
    int r = guided_pass<MLK>(b, hot, A, &areas[0].fast, sizeof(ChunkArea), open + at, cnt);
    st.guided += __popc(r & 255);
    st.heavy += __popc((r >> 8) & 255);
    if (!(r & 255) && cnt > 1) {  // levels that outgrow the items together
      const int left = r >> 16;
#pragma unroll 1
      for (int k = 0; k < cnt; ++k) {
        if ((left >> k) & 1) continue;
        r = guided_pass<MLK>(b, hot, A, &areas[0].fast, sizeof(ChunkArea), open + at + k, 1);
        st.guided += __popc(r & 255);
        st.heavy += __popc((r >> 8) & 255);
      }
    }
  }
  if (lane < 3 && (lane == 0 ? st.settled : lane == 1 ? st.guided : st.heavy))
    atomicAdd(&stats[lane], lane == 0 ? st.settled : lane == 1 ? st.guided : st.heavy);
  __syncthreads();

  if (has) write_chunk(b, hot, chunk, b.chunk, F, tag);
  // The statistics: the blocks add theirs to words that count the blocks in their upper bits,
  // and a word's last block publishes it and clears it for the next launch, so a launch of
  // this kernel alone needs nothing cleared before it.
  if (threadIdx.x < 3) {
    unsigned long long *word = ctr_ptr(b.counters, kCtrSettled) + lane;
    unsigned long long *acc = word + kStatAcc;
    const unsigned long long mine_too = (unsigned long long)stats[lane];
    const unsigned long long old = atomicAdd(acc, (1ull << kStatShift) + mine_too);
    if ((old >> kStatShift) + 1ull == (unsigned long long)gridDim.x) {
      const unsigned long long total = (old & ((1ull << kStatShift) - 1ull)) + mine_too;
      *reinterpret_cast<volatile unsigned long long *>(acc) = 0ull;
      if (b.guided == kGuidedAll) *reinterpret_cast<volatile unsigned long long *>(word) = total;
      else atomicAdd(word, total);
    }
  }
  if (b.profile && lane == 0) {
    const unsigned long long t = global_ns();
    unsigned long long *ends = ctr_ptr(b.counters, kCtrProfEnds);
    atomicMax(ends + kProfStart, ~t_enter);
    atomicMax(ends + kProfChunk, t);
    atomicAdd(ctr_ptr(b.counters, kCtrProfSums) + kProfChunk, t - t_enter);
    atomicAdd(ctr_ptr(b.counters, kCtrProfSums) + kProfSteps, 1ull);
  }
}

// The kernels of one batch: the chunk kernel (a warp per chunk) where codes of the batch
// have a guided search, the decode kernel (grid blocks) unless that leaves it nothing.
#ifndef GRAND_HOST_EMULATION
template <bool MLK>
inline cudaError_t launch_kernels(const DevBatch &b, int grid, cudaStream_t s) {
  if (b.guided) {
    const int chunks = (b.num_shots - 1) / b.chunk + 1;
    chunk_kernel<MLK><<<(chunks - 1) / kChunkWarps + 1, kChunkWarps * 32, 0, s>>>(b);
  }
  if (b.guided != kGuidedAll) decode_kernel<MLK><<<grid, kDecodeWarps * 32, 0, s>>>(b);
  return cudaGetLastError();
}
#endif

}  // namespace grand
