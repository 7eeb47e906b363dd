// Host build of the decode kernel with the guided search's tables
// (csrc/grand_guided_tables.h), for tests/test_guided_host.py: the emulation of
// host_kernels.cpp, whose own codes carry no such tables and so take the general
// path throughout, with them built as the library builds them.
//
// Usage: host_guided DIR [prep]   single-code directories of host_kernels.cpp; prints the
// same line, then the kernels that ran (enum GuidedMode) and the number of shots past
// the light budget that the guided search finished.  prep: instead, checks the tables
// that prep_kernel builds against the host's (exit code 0: equal).
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

static inline int atomicMax(int *a, int v) {
  int cur = __atomic_load_n(a, __ATOMIC_SEQ_CST);
  while (v > cur && !__atomic_compare_exchange_n(a, &cur, v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST)) {
  }
  return cur;
}
static inline int atomicMin(int *a, int v) {
  int cur = __atomic_load_n(a, __ATOMIC_SEQ_CST);
  while (v < cur && !__atomic_compare_exchange_n(a, &cur, v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST)) {
  }
  return cur;
}

#include "grand_front.cuh"
#include "grand_prep.cuh"
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

// The device-built tables of a code against the host's.
static int check_prep(const std::string &dir, const Code &k, const GuidedTables &g) {
  const std::vector<int> H = read_ints(dir + "/H.bin", (size_t)k.n * k.m);
  alignas(16) static uint32_t guided[kPrepWords], cols[kPrepMaxCols * 8], hcol[kPrepMaxCols];
  static int colw[kPrepMaxCols];
  static unsigned long long control[8] = {1, 1, 1, 1, 1, 1, 1, 1};
  DevCode tmpl = k.d, got;
  tmpl.g_gs = 0;
  tmpl.solo_branch = kSoloCpu;
  run_block(128, [&] { prep_kernel(tmpl, H.data(), cols, colw, hcol, guided, &got, control, 7); });
  bool same = control[6] == 0 && control[7] == 1;
  int most = 0, regular = 1;
  for (int c = 0; c < k.m; ++c) {
    int sum = 0;
    for (int r = 0; r < k.n; ++r) sum += H[(size_t)r * k.m + c];
    same = same && colw[c] == sum && hcol[c] == k.hcol[c];
    most = std::max(most, sum);
    regular = regular && colw[c] == colw[0];
  }
  same = same && got.max_soma == most && got.regular == regular;
  same = same && !memcmp(cols, k.cols.data(), sizeof(uint32_t) * k.cols.size());
  if (g.words.empty()) return same && got.g_gs == 0 && got.solo_branch == kSoloNone ? 0 : 5;
  const uint32_t *w = g.words.data();
  const int mw = (k.m + 31) / 32;
  same = same && got.solo_branch == kSoloCpu && got.g_gs == g.gs && got.g_deg == g.deg &&
         got.g_max_cw == g.max_cw && got.g_odd == g.odd && got.g_tab_mask == g.tab_mask;
  same = same && !memcmp(got.g_rows, w + g.o_rows, 4 * (size_t)(k.n + 1) * mw);
  same = same && !memcmp(got.g_cw, w + g.o_cw, 4 * (size_t)3 * mw);
  same = same && !memcmp(got.g_adj, w + g.o_adj, 2 * (size_t)k.n * g.deg);
  same = same && !memcmp(got.g_cols, w + g.o_cols, 4 * (size_t)k.m * g.gs);
  same = same && !memcmp(got.g_filt, w + g.o_filt, 4u << (kGuidedF - 5));
  same = same && !memcmp(got.g_hcol, w + g.o_hcol, 4 * (size_t)k.m);
  same = same && !memcmp(got.g_nib, w + g.o_nib, 4 * (size_t)nib_words(k.n));
  for (int c = 0; c < k.m && same; ++c) {  // the table: the same entries, each where a probe finds it
    uint32_t host = kNoCol, dev = kNoCol;
    for (uint32_t p = 0, i = k.hcol[c] & g.tab_mask; p <= g.tab_mask; ++p, i = (i + 1) & g.tab_mask) {
      const uint32_t a = w[g.o_tab + 2 * i + 1], b = got.g_tab[2 * i + 1];
      if ((a & 0xffffu) == (uint32_t)c) host = a;
      if (dev == kNoCol && (b & 0xffffu) == (uint32_t)c && got.g_tab[2 * i] == k.hcol[c]) dev = b;
      if ((b & 0xffffu) == kNoCol && dev == kNoCol) break;
    }
    same = host != kNoCol && host == dev;
  }
  return same ? 0 : 5;
}

int main(int argc, char **argv) {
  if (argc != 2 && argc != 3) return 2;
  const std::string dir = argv[1];
  Code k;
  if (!load_code(dir, k)) return 2;
  const GuidedTables g = build_guided_tables(k.cols, k.d.nwp, k.n, k.m, k.hcol, k.d.binary != 0, k.solo);
  if (argc == 3) return check_prep(dir, k, g);
  std::vector<uint32_t> aligned(g.words.size() + 4);
  uint32_t *base = aligned.data();
  while (reinterpret_cast<uintptr_t>(base) & 15u) ++base;
  std::copy(g.words.begin(), g.words.end(), base);
  set_guided(k.d, g, g.words.empty() ? nullptr : base);
  k.d.solo_branch = solo_branch_of(k.d);
  k.d.llr_min = *std::min_element(k.llr.begin(), k.llr.end());
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
