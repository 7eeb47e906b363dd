// grand_noalloc.cu -- grand_decode_cc_noalloc: a decode that allocates nothing.
//
// Who needs it: callers that must not allocate device memory once they are
// running -- a real-time decoding loop in a quantum-control stack that reserves
// its memory up front and may not stall in the allocator mid-experiment, or a
// host process whose device memory is already entirely owned by another
// framework's pool.  The regular entry points allocate their workspaces with
// cudaMalloc on first use (and grow them); this one keeps everything it needs
// beyond the caller's inputs and outputs in one fixed, file-scope device array.
//
// One kernel builds the code's tables on every call (grand_prep.cuh), and the batch then runs
// through the same kernels as the other entry points': the chunk kernel, then the decode
// kernel, which leaves at once when no shot is left to it.  Only the place their scratch
// lives differs: the binomial table, the packed columns and the guided search's tables, the
// code descriptor, the counters, the job table and the scratch arena are carved out of
// g_noalloc_scratch.
#include <cuda_runtime.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <mutex>

#include "grand_common.h"
#include "grand_host.h"
#include "grand_plan.h"
#include "grand_prep.cuh"

namespace grand {
namespace {

// Limits of the no-allocation path.
constexpr int kNaMaxRows = 256;                     // R <= 256 (8 words per column)
constexpr int kNaMaxCols = 1024;                    // m <= 1024
constexpr int kNaChunk = 2048;                      // shots per launch = job slots
constexpr unsigned long long kNaArenaWords = 4ull << 20;  // 16 MiB of staged search data

constexpr size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }
constexpr size_t kOffNcr = 0;
constexpr size_t kOffCode = align256(kOffNcr + sizeof(unsigned long long) * (kMaxTam + 1) * (kMaxW + 1));
constexpr size_t kOffCols = align256(kOffCode + sizeof(DevCode));
constexpr size_t kOffColw = align256(kOffCols + sizeof(uint32_t) * kNaMaxCols * 8);
constexpr size_t kOffHcol = align256(kOffColw + sizeof(int) * kNaMaxCols);
constexpr size_t kOffUpto = align256(kOffHcol + sizeof(uint32_t) * kNaMaxCols);
constexpr size_t kOffGuided = align256(kOffUpto + 8 * sizeof(unsigned long long) * (kGuidedMaxCols + 1));
constexpr size_t kOffSmall = align256(kOffGuided + sizeof(uint32_t) * kPrepWords);  // control block
constexpr size_t kOffDeferred = align256(kOffSmall + kCtlAllocBytes);
constexpr size_t kOffMap = align256(kOffDeferred + sizeof(int) * kNaChunk);     // re-run list
constexpr size_t kOffMapCount = align256(kOffMap + sizeof(int) * kNaChunk);     // its length
constexpr size_t kOffQueue = align256(kOffMapCount + 256);                       // slow queue
constexpr size_t kOffJobs = align256(kOffQueue + sizeof(unsigned long long) * kNaChunk);
constexpr size_t kOffArena = align256(kOffJobs + sizeof(Job) * kNaChunk);
constexpr size_t kScratchBytes = align256(kOffArena + sizeof(uint32_t) * kNaArenaWords);

}  // namespace

// All no-allocation calls on a device share this array; it exists for the life
// of the process on every device that loads this part of the library.  It starts
// zeroed, as the launch tags of its queue entries and Jobs require.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

namespace {

// C(n, k) by the same multiplicative formula as the host table, and their sums over k
// (DevBatch::upto).
__global__ void noalloc_ncr_kernel(unsigned long long *t, unsigned long long *upto) {
  const int n = blockIdx.x * blockDim.x + threadIdx.x;
  if (n > kMaxTam) return;
  unsigned long long sum = 0;
  for (int k = 0; k <= kMaxW; ++k) {
    unsigned long long r = 0;
    if (k <= n) {
      r = 1;
      if (k != 0 && k != n)
        for (int i = 1; i <= k; ++i) r = r * (unsigned long long)(n - i + 1) / (unsigned long long)i;
    }
    t[n * (kMaxW + 1) + k] = r;
    if (k) sum += r;
    if (n <= kGuidedMaxCols) upto[8 * n + k] = sum;
  }
  if (n <= kGuidedMaxCols) upto[8 * n + 7] = sum;
}

// One warp: the ascending list of the chunk's shots that the last round deferred
// (their heavy-shot staging did not fit the arena), and its length.  Every shot
// of the chunk had its flag written in the first round, and a re-run rewrites
// the flags of the shots it runs, so the flags are current for all cnt shots.
__global__ void noalloc_deferred_kernel(const int *deferred, int cnt, int *map, int *count) {
  const int lane = threadIdx.x & 31;
  int base = 0;
  for (int i0 = 0; i0 < cnt; i0 += 32) {
    const bool d = i0 + lane < cnt && deferred[i0 + lane] != 0;
    const unsigned bits = __ballot_sync(0xffffffffu, d);
    if (d) map[base + __popc(bits & ((1u << lane) - 1u))] = i0 + lane;
    base += __popc(bits);
  }
  if (lane == 0) *count = base;
}

// Shots that could not be searched within the arena even one at a time: a
// zero result record (found = 0), so that no stale bytes are left behind.
__global__ void noalloc_clear_kernel(const int *map, int count, GrandDecoderResult *results) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= count * 18) return;
  reinterpret_cast<uint32_t *>(results + map[i / 18])[i % 18] = 0u;
}

std::mutex g_mu;
unsigned char *g_base[64] = {};  // device address of g_noalloc_scratch per device
int g_sms[64] = {}, g_bps[64] = {};
// The status word of a round.  Where the device reaches the host's own memory (NVLink-C2C) the
// kernels raise it here, in place; otherwise in the control block, from where it is copied.
struct alignas(128) StatusWord {
  unsigned bits;
};
StatusWord g_status[64] = {};
bool g_status_here[64] = {};

}  // namespace
}  // namespace grand

using namespace grand;

extern "C" int grand_decode_cc_noalloc(const int *d_H, int n, int m, const int *d_syndromes,
                                       int num_shots, const GrandDecoderConfig *config,
                                       GrandDecoderResult *d_results, void *stream) {
  if (!config) {
    fprintf(stderr, "grand: config is NULL\n");
    return GRAND_ERR_INVALID;
  }
  const int W = config->max_error_weight;
  if (W <= 0 || W > 7) {
    fprintf(stderr, "Invalid max_error_weight: %d. Must be between 1 and 7.\n", W);
    return GRAND_ERR_INVALID;
  }
  if (num_shots < 0) {
    fprintf(stderr, "grand_decode_cc_noalloc: negative shot count\n");
    return GRAND_ERR_INVALID;
  }
  if (num_shots == 0) return 0;
  if (!d_H || !d_syndromes || !d_results) {
    fprintf(stderr, "grand_decode_cc_noalloc: NULL matrix, syndrome or result pointer\n");
    return GRAND_ERR_INVALID;
  }
  if (n <= 0 || n > kNaMaxRows || m <= 0 || m > kNaMaxCols) {
    fprintf(stderr,
            "grand_decode_cc_noalloc: H is %d x %d; this entry point supports at most %d rows and "
            "%d columns (its scratch is a fixed %zu-byte device array)\n",
            n, m, kNaMaxRows, kNaMaxCols, (size_t)kScratchBytes);
    return GRAND_ERR_LIMIT;
  }
  cudaStream_t s = (cudaStream_t)stream;
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    fprintf(stderr, "grand_decode_cc_noalloc: no usable CUDA device (%s)\n", cudaGetErrorString(e));
    return GRAND_ERR_CUDA;
  }
  unsigned char *base = nullptr;
  {
    // Set-up, once per device, with that device current: the device address of
    // the scratch array and its binomial table.
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_base[dev]) {
      void *ptr = nullptr;
      e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
      if (e != cudaSuccess) {
        fprintf(stderr, "grand_decode_cc_noalloc: cudaGetSymbolAddress failed (%s)\n",
                cudaGetErrorString(e));
        return GRAND_ERR_CUDA;
      }
      int sms = 0, bps = 0;
      e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (e == cudaSuccess) e = decode_occupancy(&bps);
      if (e == cudaSuccess) {
        noalloc_ncr_kernel<<<(kMaxTam + 256) / 256, 256, 0, s>>>(
            reinterpret_cast<unsigned long long *>((unsigned char *)ptr + kOffNcr),
            reinterpret_cast<unsigned long long *>((unsigned char *)ptr + kOffUpto));
        e = cudaGetLastError();
      }
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) {
        fprintf(stderr, "grand_decode_cc_noalloc: set-up failed (%s)\n", cudaGetErrorString(e));
        return GRAND_ERR_CUDA;
      }
      int reach = 0, atomics = 0;
      cudaDeviceGetAttribute(&reach, cudaDevAttrPageableMemoryAccess, dev);
      cudaDeviceGetAttribute(&atomics, cudaDevAttrHostNativeAtomicSupported, dev);
      g_status_here[dev] = reach && atomics;
      g_sms[dev] = sms;
      g_bps[dev] = bps > 0 ? bps : 1;
      g_base[dev] = (unsigned char *)ptr;
    }
    base = g_base[dev];
  }

  const int nw = (n + 31) / 32;
  const int nwp = nw <= 2 ? nw : (nw <= 4 ? 4 : 8);
  uint32_t *cols = reinterpret_cast<uint32_t *>(base + kOffCols);
  int *colw = reinterpret_cast<int *>(base + kOffColw);
  uint32_t *hcol = reinterpret_cast<uint32_t *>(base + kOffHcol);
  DevCode *code = reinterpret_cast<DevCode *>(base + kOffCode);

  DevCode t;
  memset(&t, 0, sizeof(t));
  t.R = n;
  t.m = m;
  t.nw = nw;
  t.nwp = nwp;
  t.mw = (m + 31) / 32;
  t.family = kCss;
  t.variant = kUniform;
  t.input_kind = kInSyndromes;
  t.W = W;
  t.Wc = W < kMaxW ? W : kMaxW;
  t.mode = config->mode_of_search;
  t.thr = config->threshold_for_hybrid;
  t.cap = config->max_size_active_positions;
  t.rec_len = n;
  t.cols = cols;
  t.colw = colw;
  t.hcol = hcol;

  {
    // whether a one-position first iteration is searched, should the code have solo columns
    DevCode x = t;
    static const int some = 0;
    x.solo_cols = &some;
    x.binary = x.max_soma = 1;
    t.solo_branch = solo_branch_of(x);
  }
  // the code's tables, on every call (nothing is kept), and the control words of the first
  // round cleared
  prep_kernel<<<1, 1024, 0, s>>>(t, d_H, cols, colw, hcol, reinterpret_cast<uint32_t *>(base + kOffGuided),
                                 code, reinterpret_cast<unsigned long long *>(base + kOffSmall),
                                 kCtlBytes / 8);
  e = cudaGetLastError();

  const Tuning &tn = tuning();
  // the decode kernel's CTAs per SM as the regular entry points choose them
  const int per_sm = decode_blocks_per_sm(g_bps[dev], tn);
  int *map = reinterpret_cast<int *>(base + kOffMap);
  int *map_count = reinterpret_cast<int *>(base + kOffMapCount);
  unsigned st = 0;       // status bits of every round of every chunk
  long long unsearched = 0;  // shots whose staging alone exceeds the arena
  for (int lo = 0; lo < num_shots && e == cudaSuccess; lo += kNaChunk) {
    const int cnt = num_shots - lo < kNaChunk ? num_shots - lo : kNaChunk;
    DevBatch b;
    memset(&b, 0, sizeof(b));
    b.num_codes = 1;
    b.codes = code;
    b.in = d_syndromes + (size_t)lo * n;
    b.results = d_results + lo;
    b.ncr = reinterpret_cast<const unsigned long long *>(base + kOffNcr);
    b.upto = reinterpret_cast<const unsigned long long *>(base + kOffUpto);
    b.jobs = reinterpret_cast<Job *>(base + kOffJobs);
    b.max_jobs = kNaChunk;
    b.counters = reinterpret_cast<unsigned long long *>(base + kOffSmall);
    b.status = g_status_here[dev] ? &g_status[dev].bits
                                  : reinterpret_cast<unsigned *>(base + kOffSmall + kStatusByteOffset);
    b.scratch = reinterpret_cast<uint32_t *>(base + kOffArena);
    b.scratch_words = kNaArenaWords;
    b.deferred = reinterpret_cast<int *>(base + kOffDeferred);
    b.queue = reinterpret_cast<unsigned long long *>(base + kOffQueue);
    b.epoch = reinterpret_cast<unsigned *>(base + kOffSmall + kCtlBytes);
    b.fast = tn.fast;
    b.light_max_log2 = tn.light_max_log2;
    b.tile_k = tn.tile_k;
    // Rounds: all of the chunk's shots, then, while some heavy shots found the
    // arena full, only those (their list built on the device), each round with
    // an empty arena.  A round in which no deferred shot fits means that each of
    // them alone needs more than the arena: those get a zero result.
    int todo = cnt;
    for (int round = 0; e == cudaSuccess; ++round) {
      b.num_shots = todo;
      b.shot_map = round == 0 ? nullptr : map;
      // The chunk kernel first where the code can have a guided search (decided on the
      // device): what that leaves is in the slow queue.  Its chunks as plan_batch's.
      b.guided = tn.fast && n <= kGuidedMaxRows ? kGuidedFirst : kGuidedNone;
      b.chunk = std::min((todo - 1) / (g_sms[dev] * kChunkMinBlocks * kChunkWarps) + 1, (int)kMaxChunk);
      // control words and status restart for every round
      if (lo > 0 || round > 0) e = cudaMemsetAsync(base + kOffSmall, 0, kCtlBytes, s);
      volatile unsigned *status = &g_status[dev].bits;
      unsigned rs = 0u;
      *status = 0u;
      if (e == cudaSuccess) e = launch_decode(b, g_sms[dev] * per_sm, s);
      if (e == cudaSuccess && !g_status_here[dev])
        e = cudaMemcpyAsync(&rs, b.status, sizeof(rs), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess) break;
      rs |= *status;
      st |= rs & ~(unsigned)(kStatusScratchOverflow | kStatusJobOverflow);
      if (!(rs & (kStatusScratchOverflow | kStatusJobOverflow))) break;
      noalloc_deferred_kernel<<<1, 32, 0, s>>>(b.deferred, cnt, map, map_count);
      int left = 0;
      e = cudaGetLastError();
      if (e == cudaSuccess)
        e = cudaMemcpyAsync(&left, map_count, sizeof(int), cudaMemcpyDeviceToHost, s);
      if (e == cudaSuccess) e = cudaStreamSynchronize(s);
      if (e != cudaSuccess || left == 0) break;
      if (left >= todo) {
        noalloc_clear_kernel<<<(left * 18 + 255) / 256, 256, 0, s>>>(map, left, b.results);
        e = cudaGetLastError();
        unsearched += left;
        break;
      }
      todo = left;
    }
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    fprintf(stderr, "grand_decode_cc_noalloc: CUDA error %s\n", cudaGetErrorString(e));
    return GRAND_ERR_CUDA;
  }
  const int rc = status_code(st);
  if (rc == GRAND_ERR_CUDA) {
    fprintf(stderr, "grand_decode_cc_noalloc: internal %s limit reached\n",
            st & kStatusCasLimit ? "ML reduction retry" : "wait");
    return rc;
  }
  if (unsearched) {
    fprintf(stderr,
            "grand_decode_cc_noalloc: %lld shot(s) need more than the fixed %llu-word search "
            "arena on their own; their results are zero (found = 0)\n",
            unsearched, kNaArenaWords);
    return GRAND_ERR_LIMIT;
  }
  if (rc == GRAND_ERR_LIMIT)
    fprintf(stderr, "grand_decode_cc_noalloc: an active-position set exceeded %d\n", kMaxTam);
  return rc;
}
