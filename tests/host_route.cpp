// Host build of both decoding kernels, planned as the library plans a batch (csrc/grand_plan.h):
// the emulation of host_kernels.cpp with the codes' guided tables and their one-position rule
// set, for tests/test_route_host.py.
//
// Usage: host_route DIR [tables=0]   a directory of host_kernels.cpp's mixed form (any number of
// codes; DEM records are detectors and then logical flips); writes res.bin and prints that
// program's line, then the plan and what became of the shots.  tables=0: codes without guided
// tables, so the decode kernel alone.
#include <sys/mman.h>

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
#include "grand_plan.h"

// The last block of a batch of the most shots that an int counts, in address space that only
// its records and results occupy.
static int run_edge(const std::string &dir, DevBatch &b, const DevCode &cd, const std::vector<int> &rec) {
  const size_t all = 0x7fffffff, count = rec.size() / cd.rec_len;
  auto space = [](size_t bytes) {
    return (char *)mmap(nullptr, bytes, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
  };
  char *in = space(all * cd.rec_len * 4), *out = space(all * sizeof(GrandDecoderResult));
  if (in == MAP_FAILED || out == MAP_FAILED) return 7;
  memcpy(in + (all - count) * cd.rec_len * 4, rec.data(), 4 * rec.size());
  b.in = (const int *)in;
  b.results = (GrandDecoderResult *)out;
  b.in_off = nullptr;
  b.shot_code = nullptr;
  b.num_codes = 1;
  b.num_shots = (int)all;
  plan_batch(b, &cd, 1, 152, true);
  if (b.guided != kGuidedAll) return 8;
  b.chunk = 27;  // (one that does not divide the batch)
  gridDim.x = (unsigned)(((all - 1) / b.chunk) / kChunkWarps + 1);
  blockIdx.x = gridDim.x - 1;
  run_block(kChunkWarps * 32, [&] { chunk_kernel<false>(b); });
  if (*b.status) return 4;
  write_bytes(dir + "/res.bin", out + (all - count) * sizeof(GrandDecoderResult), sizeof(GrandDecoderResult) * count);
  return 0;
}

int main(int argc, char **argv) {
  if (argc < 2) return 2;
  const std::string dir = argv[1];
  const bool tables = !(argc > 2 && !strcmp(argv[2], "tables=0"));
  int K, N, light, tile_k;
  FILE *mf = fopen((dir + "/mixed.txt").c_str(), "r");
  if (!mf || fscanf(mf, "%d %d %d %d", &K, &N, &light, &tile_k) != 4) return 2;
  fclose(mf);
  std::vector<Code> codes(K);
  std::vector<DevCode> dcs(K);
  std::vector<std::vector<uint32_t>> blocks(K);
  for (int k = 0; k < K; ++k) {
    Code &c = codes[k];
    if (!load_code(dir + "/code" + std::to_string(k), c)) return 2;
    if (c.family == kDem) c.d.rec_len = c.n + c.nl;
    if (tables) {
      const GuidedTables g = build_guided_tables(c.cols, c.d.nwp, c.n, c.m, c.hcol, c.d.binary != 0, c.solo);
      blocks[k].resize(g.words.size() + 4);
      uint32_t *base = blocks[k].data();
      while (reinterpret_cast<uintptr_t>(base) & 15u) ++base;
      std::copy(g.words.begin(), g.words.end(), base);
      set_guided(c.d, g, g.words.empty() ? nullptr : base);
    }
    c.d.solo_branch = solo_branch_of(c.d);
    c.d.llr_min = *std::min_element(c.llr.begin(), c.llr.end());
    dcs[k] = c.d;
  }
  FILE *rf = fopen((dir + "/rec.bin").c_str(), "rb");
  if (!rf) return 2;
  fseek(rf, 0, SEEK_END);
  const size_t total = (size_t)ftell(rf) / 4;
  fclose(rf);
  const std::vector<int> rec = read_ints(dir + "/rec.bin", total);
  std::vector<long long> off(N);
  FILE *of = fopen((dir + "/off.bin").c_str(), "rb");
  if (!of || fread(off.data(), 8, N, of) != (size_t)N) return 2;
  fclose(of);
  const std::vector<int> shot_code = read_ints(dir + "/code.bin", N);
  std::vector<GrandDecoderResult> res(N);

  std::vector<unsigned long long> ncr((size_t)(kMaxTam + 1) * (kMaxW + 1));
  for (int a = 0; a <= kMaxTam; ++a)
    for (int k = 0; k <= kMaxW; ++k) ncr[(size_t)a * (kMaxW + 1) + k] = C(a, k);
  std::vector<unsigned long long> upto(8 * (kGuidedMaxCols + 1), 0ull);
  for (int n = 0; n <= kGuidedMaxCols; ++n)
    for (int k = 1; k < 8; ++k)
      upto[8 * (size_t)n + k] = upto[8 * (size_t)n + k - 1] + (k <= kMaxW ? C(n, k) : 0ull);
  std::vector<Job> jobs(N);
  alignas(128) static unsigned long long small[kCtlAllocBytes / 8];
  std::vector<uint32_t> scratch(8u << 20), rec_cache((size_t)N * kRecCacheWords, 0xa5a5a5a5u);
  std::vector<int> deferred(N, 0);
  std::vector<unsigned long long> queue(N, 0ull);

  DevBatch b;
  memset(&b, 0, sizeof(b));
  b.num_shots = N;
  b.num_codes = K;
  b.codes = dcs.data();
  b.in = rec.data();
  b.in_off = off.data();
  b.shot_code = shot_code.data();
  b.results = res.data();
  b.ncr = ncr.data();
  b.upto = upto.data();
  b.jobs = jobs.data();
  b.max_jobs = N;
  b.counters = small;
  b.status = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(small) + kStatusByteOffset);
  b.scratch = scratch.data();
  b.scratch_words = scratch.size();
  b.deferred = deferred.data();
  b.queue = queue.data();
  b.rec_cache = rec_cache.data();
  b.epoch = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(small) + kCtlBytes);
  b.fast = 1;
  b.light_max_log2 = light;
  b.tile_k = tile_k;
  if (argc > 2 && !strcmp(argv[2], "edge")) return run_edge(dir, b, dcs[0], rec);
  plan_batch(b, dcs.data(), K, 1, true);
  if (b.guided) {
    gridDim.x = (unsigned)(((N - 1) / b.chunk) / kChunkWarps + 1);
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
    if (d) return 3;
  const unsigned slow = (unsigned)(*ctr_ptr(small, kCtrChunks) & 0xffffffffull);
  int cached = 0;
  for (unsigned i = 0; i < slow; ++i) cached += (queue[i] >> 31) & 1u;
  const unsigned long long *stat = ctr_ptr(small, kCtrSettled);
  printf("ok %d shots, %llu jobs, %llu slow, status %u\n", N, *ctr_ptr(small, kCtrJobs) >> 40,
         *ctr_ptr(small, kCtrSlowDone), *b.status);
  printf("guided %d chunk %d settled %llu searched %llu heavy %llu cached %d\n", b.guided, b.chunk,
         stat[0], stat[1], stat[2], cached);
  if (*b.status) return 4;
  write_bytes(dir + "/res.bin", res.data(), sizeof(GrandDecoderResult) * N);
  return 0;
}
