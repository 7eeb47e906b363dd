// Host build of the decode kernel with the guided search's tables
// (csrc/grand_guided_tables.h), for tests/test_guided_host.py: the emulation of
// host_kernels.cpp, whose own codes carry no such tables and so take the general
// path throughout, with them built as the library builds them.
//
// Usage: host_guided DIR   single-code directories of host_kernels.cpp; prints the
// same line, then the kernels that ran (enum GuidedMode) and the number of shots past
// the light budget that the guided search finished.
#define main host_kernels_main
#include "host_kernels.cpp"
#undef main

// the block's threads meet; shared-memory atomics
static std::atomic<int> g_block_count{0}, g_block_gen{0};
static void __syncthreads() {
  const int gen = g_block_gen.load();
  if (g_block_count.fetch_add(1) + 1 == (int)blockDim.x) {
    g_block_count.store(0);
    g_block_gen.fetch_add(1);
    return;
  }
  while (g_block_gen.load() == gen) std::this_thread::yield();
}
static inline int atomicAdd(int *a, int v) { return __atomic_fetch_add(a, v, __ATOMIC_SEQ_CST); }

#include "grand_front.cuh"
#include "grand_guided_tables.h"

// The kernels of a batch as the library launches them (launch_kernels).
static void run_guided_batch(DevBatch &b, int N) {
  std::vector<unsigned long long> ncr((size_t)(kMaxTam + 1) * (kMaxW + 1));
  for (int a = 0; a <= kMaxTam; ++a)
    for (int k = 0; k <= kMaxW; ++k) ncr[(size_t)a * (kMaxW + 1) + k] = C(a, k);
  std::vector<Job> jobs(N);
  alignas(128) static unsigned long long small[kCtlAllocBytes / 8];
  const unsigned long long scratch_words = 8ull << 20;
  std::vector<uint32_t> scratch(scratch_words);
  std::vector<int> deferred(N, 0);
  std::vector<unsigned long long> queue(N, 0ull);
  std::vector<uint32_t> rec_cache((size_t)N * kRecCacheWords, 0xa5a5a5a5u);
  b.num_shots = N;
  b.ncr = ncr.data();
  std::vector<unsigned long long> upto(8 * (kGuidedMaxCols + 1), 0ull);
  for (int n = 0; n <= kGuidedMaxCols; ++n)
    for (int k = 1; k < 8; ++k)
      upto[8 * (size_t)n + k] = upto[8 * (size_t)n + k - 1] + (k <= kMaxW ? C(n, k) : 0ull);
  b.upto = upto.data();
  b.jobs = jobs.data();
  b.max_jobs = N;
  b.counters = small;
  b.status = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(small) + kStatusByteOffset);
  b.scratch = scratch.data();
  b.scratch_words = scratch_words;
  b.deferred = deferred.data();
  b.queue = queue.data();
  b.rec_cache = rec_cache.data();
  b.epoch = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(small) + kCtlBytes);
  if (b.guided) {
    const int chunks = (N - 1) / b.chunk + 1;
    gridDim.x = (unsigned)((chunks - 1) / kChunkWarps + 1);
    for (blockIdx.x = 0; blockIdx.x < gridDim.x; ++blockIdx.x)
      run_block(kChunkWarps * 32, [&] {
        if (b.has_ml) chunk_kernel<true>(b);
        else chunk_kernel<false>(b);
      });
    blockIdx.x = 0;
    gridDim.x = 1;
  }
  if (b.guided != kGuidedAll)
    run_block(kDecodeWarps * 32, [&] {
      if (b.has_ml) decode_kernel<true>(b);
      else decode_kernel<false>(b);
    });
  for (int d : deferred)
    if (d) exit(3);
  printf("ok %d shots, %llu jobs, %llu slow, status %u\n", N, *ctr_ptr(small, kCtrJobs) >> 40,
         *ctr_ptr(small, kCtrSlowDone), *b.status);
  if (*b.status) exit(4);
}

int main(int argc, char **argv) {
  if (argc != 2) return 2;
  const std::string dir = argv[1];
  Code k;
  if (!load_code(dir, k)) return 2;
  const GuidedTables g = build_guided_tables(k.cols, k.d.nwp, k.n, k.m, k.hcol, k.d.binary != 0, k.solo);
  std::vector<uint32_t> aligned(g.words.size() + 4);
  uint32_t *base = aligned.data();
  while (reinterpret_cast<uintptr_t>(base) & 15u) ++base;
  std::copy(g.words.begin(), g.words.end(), base);
  set_guided(k.d, g, g.words.empty() ? nullptr : base);
  k.d.solo_branch = solo_branch_of(k.d);
  const int N = k.N, m = k.m, nl = k.nl;
  const bool dem = k.family == kDem;
  const std::vector<int> rec = read_ints(dir + "/rec.bin", (size_t)N * k.rec_len);
  const std::vector<int> logicals =
      dem ? read_ints(dir + "/log.bin", (size_t)N * std::max(k.log_len, 1)) : std::vector<int>();
  std::vector<GrandDecoderResult> res(N);
  std::vector<unsigned char> dec((size_t)N * m, 7), declog((size_t)N * std::max(nl, 1), 7);
  std::vector<float> cost(N, -1.0f);
  DevBatch b;
  memset(&b, 0, sizeof(b));
  b.num_codes = 1;
  b.codes = &k.d;
  b.in = rec.data();
  b.results = res.data();
  b.dec_err = dec.data();
  if (dem) {
    b.in_log = logicals.data();
    b.dec_log = declog.data();
    b.ml_cost = k.variant == kMl ? cost.data() : nullptr;
  }
  b.light_max_log2 = k.light;
  b.tile_k = k.tile_k;
  b.has_ml = k.variant == kMl;
  const char *fe = getenv("GRAND_EMU_FAST");
  b.fast = (fe && *fe == '0') ? 0 : 1;
  b.guided = !k.d.g_gs || !b.fast ? kGuidedNone : (guided_closed(k.d) ? kGuidedAll : kGuidedFirst);
  b.chunk = 1 + N % kMaxChunk;
  run_guided_batch(b, N);
  printf("guided %d heavy %llu\n", b.guided, ctr_ptr(b.counters, kCtrSettled)[2]);
  write_bytes(dir + "/res.bin", res.data(), sizeof(GrandDecoderResult) * N);
  write_bytes(dir + "/dec.bin", dec.data(), dec.size());
  if (dem) {
    write_bytes(dir + "/declog.bin", declog.data(), (size_t)N * nl);
    write_bytes(dir + "/cost.bin", cost.data(), sizeof(float) * N);
  }
  return 0;
}
