// grand_chunk.cuh -- the chunk step of a decoding launch (sm_103a), and the chunk kernel
// that runs it with the guided search.
//
// classify_chunk (up to kMaxChunk launch slots, one lane per shot)
//   packs the shots' records with coalesced ballots, forms each syndrome and
//   settles the common shots outright: an empty syndrome (grand_decoder.cu:1223-1241),
//   and a first threshold iteration with one active position whose column equals
//   the syndrome (weight-1 match, 1 candidate tested).
//
// chunk_kernel
//   takes the remaining shots of a chunk one after another through the guided search
//   (grand_guided.cuh), by the warp that holds their syndromes and record bits.  One
//   warp per chunk, blocks scheduled by the hardware: nothing waits.  It is a kernel of
//   its own, not a step of the persistent decode kernel, for its working set: there
//   (46 KB of shared memory per block, 128 registers, 650 KB of code) the same search
//   ran at 16 warps per SM out of 28 KB of L1 and missed the instruction caches
//   (headline 80 us, mix 178 us, noisy [[288]] 164 us); here 48, 125 and 92 us.
#pragma once

#include "grand_guided.cuh"
#include "grand_kernels.cuh"

namespace grand {

// ---------------------------------------------------------------------------
// Chunks of up to kMaxChunk launch slots, one lane per shot.
// ---------------------------------------------------------------------------
constexpr int kFastWords = 8;         // syndrome words of a lane's shot (R <= 256)
constexpr int kFastLogWords = 4;      // DEM logical words (n_logicos <= 128)
constexpr int kFastErrWords = 32;     // error-record words (m <= 1024)
constexpr int kFastLogBallots = kMaxChunk * kFastLogWords;  // ballot words of separate logical entries

// classify_chunk's part of a warp's shared memory.  A shot's row holds its syndrome
// (words 0 .. 7), sketch (8), supplied weight (9) and logical words (10 .. 13) while it is open, and its result's 18 words once it is settled.
struct FastArea {
  uint32_t bits[kFastBallots + 8];      // the run's records, entry after entry (flat_ballots)
  uint32_t lbits[kFastLogBallots + 8];  // the same for DEM logicals kept in their own array
  uint32_t row[kMaxChunk][18];
  int shot[kMaxChunk];
};
constexpr int kRowSketch = kFastWords, kRowWeight = kFastWords + 1, kRowLog = kFastWords + 2;
static_assert(kRowLog + kFastLogWords <= 18, "an open shot's words fit its row");
static_assert(sizeof(FastArea) <= sizeof(WarpArea), "FastArea must fit the decode kernel's area");

// The chunk kernel's shared memory of one warp.
struct ChunkArea {
  GuidedArea guided;
  FastArea fast;
  DevCode code;  // the code being searched
};

// The nonzero flags of the n entries at p as a bit vector: entry e is bit pad + e, with
// pad (returned, 0 .. 3) the entries between p and the 16-byte boundary below it; other
// bits are arbitrary.  Lanes read four entries at a time, eight 16-byte loads each in
// flight (records read in place from host memory need the bytes in flight), kept out of
// L1; two lanes' flags make a byte.  The groups of four that p and the end cut are
// read entry by entry.  Writes whole rows of 128 entries (16 bytes).
static __device__ __noinline__ int flat_ballots(const int *p, int n, uint32_t *bits) {
  const int lane = threadIdx.x & 31;
  const int pad = (int)((reinterpret_cast<uintptr_t>(p) >> 2) & 3u);
  p -= pad;
  n += pad;
  uint8_t *bytes = reinterpret_cast<uint8_t *>(bits);
  const int4 *p4 = reinterpret_cast<const int4 *>(p);
  const int first = pad ? 1 : 0, full = n >> 2;  // whole groups: first .. full - 1
#pragma unroll 1
  for (int r0 = 0; r0 * 128 < n; r0 += 8) {
    int4 v[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int i = (r0 + u) * 32 + lane;
      v[u] = i >= first && i < full ? __ldcg(p4 + i) : make_int4(0, 0, 0, 0);
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      if ((r0 + u) * 128 < n) {
        const unsigned nib = (v[u].x ? 1u : 0u) | (v[u].y ? 2u : 0u) | (v[u].z ? 4u : 0u) | (v[u].w ? 8u : 0u);
        const unsigned next = __shfl_down_sync(kFull, nib, 1);
        if (!(lane & 1)) bytes[((r0 + u) * 32 + lane) >> 1] = (uint8_t)(nib | (next << 4));
      }
    }
  }
  if (pad | (n & 3)) {
    __syncwarp();
    if (lane == 0) {
#pragma unroll 1
      for (int e = pad; e < n; ++e) {
        if (e >= 4 * first && e < 4 * full) e = 4 * full;
        if (e < n && __ldcg(p + e)) bytes[e >> 3] |= (uint8_t)(1u << (e & 7));
      }
    }
  }
  return pad;
}

// Word q of the nbits-entry bit vector that starts at entry `off` of a flat
// ballot array (entries past nbits masked off).
__device__ __forceinline__ uint32_t flat_word(const uint32_t *bits, int off, int q, int nbits) {
  const int e = off + 32 * q;
  uint32_t w = __funnelshift_r(bits[e >> 5], bits[(e >> 5) + 1], e & 31);
  const int rem = nbits - 32 * q;
  if (rem < 32) w &= (1u << rem) - 1u;
  return w;
}

// Statistics of a warp, added to the control block when it leaves: shots settled without
// a search, by the guided search, and those of the latter past the light budget.
struct ChunkStats {
  int settled, guided, heavy;
};
__device__ __forceinline__ void add_stats(const DevBatch &b, const ChunkStats &st) {
  unsigned long long *w = ctr_ptr(b.counters, kCtrSettled);
  if (st.settled) atomicAdd(w, (unsigned long long)st.settled);
  if (st.guided) atomicAdd(w + 1, (unsigned long long)st.guided);
  if (st.heavy) atomicAdd(w + 2, (unsigned long long)st.heavy);
}

// Settles the shots of launch slots size * chunk + [0, size), size <= kMaxChunk.
//
// One lane per shot forms the syndromes and settles the shots that need no search: an
// empty syndrome, or a first iteration with one active position whose column equals
// the syndrome.  The results are exactly those of the general path: the one position
// is the only candidate of the iteration (found at weight 1, rank 0; one candidate
// counted on either branch, hibrido 0 / -1), and its active set is the set of nonzero
// columns contained in the syndrome (flagged-check count = column weight, for
// 0/1 matrices regular or not), a solo column found by the syndrome's sketch.
//
// GUIDED: the warp then takes the other shots one after another through the guided
// search, from the syndromes and record bits it holds (area: the warp's search area
// and code copy).  What is left -- codes without the search's tables, records too wide
// for a lane, levels that do not fit -- is appended to the slow queue with tag (the
// launch epoch + 1).
//
// kCtrChunks counts the chunks done (high half) and the queue entries reserved (low
// half) in one word, so that a warp that sees every chunk done sees every
// reservation too, with no fence in between.
template <bool MLK, bool GUIDED>
__device__ __forceinline__ void classify_chunk(const DevBatch &b, int chunk, int size, FastArea &F,
                                               ChunkArea *area, ChunkStats &st, unsigned tag) {
  const int lane = threadIdx.x & 31;
  const int slot = chunk * size + lane;
  const bool valid = lane < size && slot < b.num_shots;
  const unsigned long long t_start = global_ns();
  unsigned long long tp = b.profile ? t_start : 0ull;
  const int shot = valid ? (b.shot_map ? b.shot_map[slot] : slot) : 0;
  const int ci = (valid && b.shot_code) ? b.shot_code[shot] : 0;
  const DevCode &cd = b.codes[ci];
  const bool errs = cd.input_kind == kInErrors;
  const bool dem = cd.family == kDem;
  const bool packed = cd.packed != 0;
  const int nw = cd.nw;
  const int nbits = errs ? cd.m : cd.R;       // entries of the record's leading bit vector
  const int nwords = (nbits + 31) >> 5;
  bool ok = valid && nw <= kFastWords && (!errs || nwords <= kFastErrWords) &&
            (!dem || cd.nlw <= kFastLogWords);
  const long long rbase = valid ? (b.in_off ? b.in_off[shot] : (long long)shot * cd.rec_len) : 0;
  uint32_t *row = F.row[valid ? lane : 0];
  if (valid) F.shot[lane] = shot;

  // ---- the records: int32 entries through coalesced ballots over runs of
  //      back-to-back records, bit-packed words read directly ------------------
  int ow = 0, epos = -1;
  uint32_t hs = 0u;
  bool log_ok = true;
  const bool sep = b.in_log != nullptr;
  int lpad = 0;
  if (sep) {
    // the chunk's logicals lie back to back unless the shots are mapped (a single-code
    // call: every lane has the same code)
    log_ok = !b.shot_map && !packed && b.num_codes == 1;
    if (__any_sync(kFull, ok && dem && log_ok)) {
      const int first = chunk * size;
      const int cnt = b.num_shots - first < size ? b.num_shots - first : size;
      lpad = flat_ballots(b.in_log + (long long)first * cd.n_logicos, cnt * cd.n_logicos, F.lbits);
      __syncwarp();
    }
  }
  const uint32_t *cols = cd.g_gs ? cd.g_cols : cd.cols;
  const uint32_t *hcol = cd.g_gs ? cd.g_hcol : cd.hcol;
  const int stride = cd.g_gs ? cd.g_gs : cd.nwp;  // words per column
  // this lane's record out of ballots of the entries from `first` on (or its packed words)
  auto take = [&](int at, const uint32_t *rw) {
    auto word = [&](int q) {
      if (!rw) return flat_word(F.bits, at, q, nbits);
      const uint32_t w = __ldcg(rw + q);
      const int rem = nbits - 32 * q;
      return rem < 32 ? w & ((1u << rem) - 1u) : w;
    };
    if (errs) {
      Resid s;
      s.a = s.b = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 1
      for (int q = 0; q < nwords; ++q) {
        uint32_t w = word(q);
        ow += __popc(w);
#pragma unroll 1
        for (; w; w &= w - 1u) {
          const int c = q * 32 + __ffs((int)w) - 1;
          epos = c;
          hs ^= __ldg(hcol + c);
          if (stride >= 4) {
            xor_col(cols, stride == 8, (unsigned)c, s);
          } else {
            s.a.x ^= __ldg(cols + c * stride);
            if (stride == 2) s.a.y ^= __ldg(cols + c * 2 + 1);
          }
        }
      }
      row[0] = s.a.x;
      row[1] = s.a.y;
      row[2] = s.a.z;
      row[3] = s.a.w;
      row[4] = s.b.x;
      row[5] = s.b.y;
      row[6] = s.b.z;
      row[7] = s.b.w;
    } else {
#pragma unroll 1
      for (int k = 0; k < kFastWords; ++k) {
        uint32_t w = k < nw ? word(k) : 0u;
        row[k] = w;
#pragma unroll 1
        for (; w; w &= w - 1u) hs ^= row_hash(k * 32 + __ffs((int)w) - 1);
      }
      if (dem) {
        const uint32_t *lw = rw ? (sep ? reinterpret_cast<const uint32_t *>(b.in_log) + (size_t)shot * cd.nlw
                                       : rw + nw)
                                : nullptr;
#pragma unroll 1
        for (int k = 0; k < kFastLogWords; ++k) {
          const int rem = cd.n_logicos - 32 * k;
          uint32_t w = 0u;
          if (k < cd.nlw) {
            if (lw) w = __ldcg(lw + k) & (rem < 32 ? (1u << rem) - 1u : kFull);
            else if (sep) w = flat_word(F.lbits, lpad + lane * cd.n_logicos, k, cd.n_logicos);
            else w = flat_word(F.bits, at + cd.R, k, cd.n_logicos);
          }
          row[kRowLog + k] = w;
        }
      }
    }
    row[kRowSketch] = hs;
    row[kRowWeight] = (uint32_t)ow;
  };
  ok = ok && (packed || !dem || log_ok || !sep);
  // Runs of consecutive lanes whose int32 records lie back to back (one run for a
  // batch packed in slot order; a few where requests' records sit in separate
  // buffers): each run's entries through one pass of ballots.
  const int rlen = dem && !sep ? cd.R + cd.n_logicos : nbits;
  const bool mine = valid && !packed;
  const long long pend = __shfl_up_sync(kFull, rbase + rlen, 1);
  const bool pint = __shfl_up_sync(kFull, mine ? 1 : 0, 1) != 0;
  const unsigned members_all = __ballot_sync(kFull, mine);
  const unsigned all_starts = __ballot_sync(kFull, mine && (lane == 0 || !pint || pend != rbase));
  const bool one_run = (all_starts & (all_starts - 1u)) == 0u;
  int at = 0;  // where this lane's record starts in the ballots
  unsigned starts = all_starts;
  bool words = __any_sync(kFull, ok && packed);  // packed records still to be taken
#pragma unroll 1
  while (starts || words) {
    bool in_run = packed;
    const uint32_t *rw = nullptr;
    if (starts) {
      const int l0 = __ffs((int)starts) - 1;
      starts &= starts - 1u;
      const int lnext = starts ? __ffs((int)starts) - 1 : 32;
      const unsigned span = (lnext == 32 ? kFull : ((1u << lnext) - 1u)) & ~((1u << l0) - 1u);
      const unsigned members = members_all & span;  // l0 .. the run's last lane, no gaps
      const long long first = __shfl_sync(kFull, rbase, l0);
      const long long end = __shfl_sync(kFull, rbase + rlen, 31 - __clz((int)members));
      in_run = (members >> lane) & 1u;
      if (end - first > 32ll * kFastBallots) {
        if (in_run) ok = false;  // longer than the chunk's ballot area: slow path
        continue;
      }
      const int pad = flat_ballots(b.in + first, (int)(end - first), F.bits);
      __syncwarp();
      at = in_run ? (int)(rbase - first) + pad : at;
    } else {
      words = false;
      rw = reinterpret_cast<const uint32_t *>(b.in) + rbase;
    }
    if (in_run && ok) take(at, rw);
    __syncwarp();  // every lane has read the run's bits before the next run's
  }
  tp = prof_lap(b, kProfChunkRead, tp);

  // ---- settle: empty syndrome, or a one-position first iteration matched ----
  bool empty = ok;
#pragma unroll 1
  for (int k = 0; k < nw && empty; ++k) empty = row[k] == 0u;
  bool found = false;
  int pos = -1, deg = 0, iseq = 0;
  if (ok && !empty && cd.solo_branch) {
    // the first iteration's active set is the nonzero columns contained in s:
    // it is one column whose only candidate matches exactly when s equals a
    // solo column, found by s's sketch (in the guided search's table, or in one of the
    // solo columns alone)
    const uint32_t mask = cd.g_gs ? cd.g_tab_mask : cd.solo_mask;
    uint32_t i = hs & mask;
#pragma unroll 1
    for (uint32_t probe = 0; probe <= mask && !found; ++probe) {
      uint2 e;
      if (cd.g_gs) e = __ldg(reinterpret_cast<const uint2 *>(cd.g_tab) + i);
      else e = make_uint2(__ldg(cd.solo_keys + i), (unsigned)__ldg(cd.solo_cols + i) | kSoloFlag);
      const int c = (int)(e.y & 0xffffu);
      if (c == (int)kNoCol) break;
      if (e.x == hs && (e.y & kSoloFlag)) {
        bool eq = true;
#pragma unroll 1
        for (int k = 0; k < nw && eq; ++k) eq = __ldg(cols + c * stride + k) == row[k];
        if (eq) {
          found = true;
          pos = c;
        }
      }
      i = (i + 1u) & mask;
    }
    if (found) {
      if (!dem && errs) {
        iseq = (ow == 1 && epos == pos) ? 1 : 0;
        deg = 1;
        found = iseq != 0;  // a different supplied error needs the degeneracy test
      } else if (dem) {
        deg = 1;
#pragma unroll 1
        for (int k = 0; k < cd.nlw; ++k)
          if (__ldg(cd.lcols + (size_t)pos * cd.nlw + k) != row[kRowLog + k]) deg = 0;
      }
    }
  }
  const bool done = empty || found;
  if (!found) pos = -1;
  const unsigned settled = __ballot_sync(kFull, done);
  st.settled += __popc(settled);
  tp = prof_lap(b, kProfChunkTest, tp);

  // ---- results of the settled shots ----------------------------------------
  if (settled) {
    if (done) {
      const unsigned long long now = global_ns();
#pragma unroll
      for (int w = 0; w < 18; ++w) row[w] = 0u;
      row[2] = (uint32_t)ow;
      if (empty) {
        row[8] = (uint32_t)-2;
      } else {
        // the times: counts and search half each, and the whole
        const unsigned long long dt = now - t_start;
        const unsigned long long h = (unsigned long long)__double_as_longlong(1e-6 * (double)(dt >> 1));
        const unsigned long long t = (unsigned long long)__double_as_longlong(1e-6 * (double)dt);
        row[10] = row[12] = (uint32_t)h;
        row[11] = row[13] = (uint32_t)(h >> 32);
        row[16] = (uint32_t)t;
        row[17] = (uint32_t)(t >> 32);
        row[0] = 1u;
        row[1] = 1u;
        row[3] = (uint32_t)deg;
        row[4] = (uint32_t)iseq;
        row[5] = 1u;
        row[6] = 1u;
        row[8] = cd.solo_branch == kSoloGpu ? 0u : (uint32_t)-1;
        row[9] = 1u;
      }
      if (b.ml_cost)
        b.ml_cost[shot] = MLK && found && cd.variant == kMl ? __fadd_rn(0.0f, __ldg(cd.llr + pos)) : 0.0f;
      if (b.deferred) b.deferred[shot] = 0;
    }
    __syncwarp();
    // one coalesced pass over the rows: word i belongs to lane i / 18's shot
#pragma unroll 1
    for (int i = lane; i < size * 18; i += 32) {
      const int j = (i * 3641) >> 16;  // i / 18 for i < 18 * kMaxChunk
      if ((settled >> j) & 1u)
        reinterpret_cast<uint32_t *>(b.results + F.shot[j])[i - 18 * j] = F.row[j][i - 18 * j];
    }
    if (b.dec_err || b.dec_log) {
#pragma unroll 1
      for (unsigned mm = settled; mm; mm &= mm - 1u) {
        const int j = __ffs((int)mm) - 1;
        const int sj = F.shot[j];
        const int cj = __shfl_sync(kFull, ci, j);
        const int pj = __shfl_sync(kFull, pos, j);
        const DevCode &cdj = b.codes[cj];
        if (b.dec_err)
          bits_to_bytes(b.dec_err + (size_t)sj * cdj.m, cdj.m,
                        pj >= 0 && (pj >> 5) == lane ? 1u << (pj & 31) : 0u);
        if (b.dec_log && cdj.family == kDem)
          bits_to_bytes(b.dec_log + (size_t)sj * cdj.n_logicos, cdj.n_logicos,
                        pj >= 0 && lane < cdj.nlw ? __ldg(cdj.lcols + (size_t)pj * cdj.nlw + lane) : 0u);
      }
    }
  }
  tp = prof_lap(b, kProfChunkWrite, tp);

  unsigned slow = __ballot_sync(kFull, valid && !done);

  // ---- the others: the guided search ------------------------------------------
  if constexpr (GUIDED) {
    DevCode &code = area->code;
    int loaded = -1;
#pragma unroll 1
    for (unsigned mm = __ballot_sync(kFull, ok && !done && cd.g_gs); mm; mm &= mm - 1u) {
      const int j = __ffs((int)mm) - 1;
      const int cj = __shfl_sync(kFull, ci, j);
      int at_j = __shfl_sync(kFull, at, j);
      const long long rb_j = __shfl_sync(kFull, rbase, j);
      if (loaded != cj) {
        load_code(code, b.codes + cj);
        loaded = cj;
      }
      const uint32_t *rj = F.row[j];
      uint32_t eb = 0u;
      if (code.family == kDem) {
        if (lane < code.nlw) eb = rj[kRowLog + lane];
      } else if (code.input_kind == kInErrors) {
        if (!code.packed && !one_run) {  // a later run took its bits' place
          at_j = flat_ballots(b.in + rb_j, code.m, F.bits);
          __syncwarp();
        }
        const int rem = code.m - 32 * lane;
        if (rem > 0)
          eb = code.packed ? __ldcg(reinterpret_cast<const uint32_t *>(b.in) + rb_j + lane) &
                                 (rem < 32 ? (1u << rem) - 1u : kFull)
                           : flat_word(F.bits, at_j, lane, code.m);
      }
      const int r = guided_shot<MLK>(b, code, F.shot[j], area->guided, lane < kFastWords ? rj[lane] : 0u,
                                     rj[kRowSketch], eb, (int)rj[kRowWeight], global_ns());
      if (r) {
        slow &= ~(1u << j);
        ++st.guided;
        st.heavy += r - 1;
      }
    }
    if (b.guided == kGuidedAll) {
      if (slow && lane == 0) atomicOr(b.status, kStatusWaitLimit);  // never: see guided_closed
      return;
    }
  }

  // ---- what is left: the slow queue -------------------------------------------
  unsigned long long base = 0;
  if (lane == 0)
    base = atomicAdd(ctr_ptr(b.counters, kCtrChunks), (1ull << 32) + (unsigned long long)__popc(slow));
  if (slow) {
    base = __shfl_sync(kFull, base, 0) & 0xffffffffull;
    if ((slow >> lane) & 1u) {
      // its record's bits for the per-shot path, in place of a second read of the caller's
      const bool cache = b.rec_cache && ok && !packed && one_run &&
                         nwords + (dem ? cd.nlw : 0) <= kRecCacheWords;
      if (cache) {
        uint32_t *cp = b.rec_cache + (size_t)slot * kRecCacheWords;
#pragma unroll 1
        for (int q = 0; q < nwords; ++q) cp[q] = flat_word(F.bits, at, q, nbits);
#pragma unroll 1
        for (int k = 0; k < cd.nlw && dem; ++k) cp[nwords + k] = row[kRowLog + k];
      }
      // the entry carries this launch's tag: a ticket holder that reads it knows it
      // is not a leftover of an earlier launch
      *reinterpret_cast<volatile unsigned long long *>(b.queue + base + __popc(slow & ((1u << lane) - 1u))) =
          ((unsigned long long)tag << 32) | (unsigned)slot | (cache ? 0x80000000u : 0u);
    }
  }
  __syncwarp();
}

// A load whose value nothing uses, for the line it brings into L1.
__device__ __forceinline__ void touch_line(const void *p) {
#ifdef GRAND_HOST_EMULATION
  (void)p;
#else
  unsigned x;
  asm volatile("ld.global.nc.u32 %0, [%1];" : "=r"(x) : "l"(p));
#endif
}
constexpr int kWarmCodes = 8;   // codes whose tables are fetched ahead (about 60 KB for the BB codes)
constexpr int kWarmTam = 192;   // active sets whose binomials are

// One warp per chunk of the batch.
constexpr int kChunkWarps = 4;
// Resident blocks per SM: 5 leave a thread 96 registers and the SM about 130 KB of L1.
// Measured (4 / 5 / 6 / 8 blocks): headline batch 47.8 / 48.4 / 52.2 / 59.2 us, noisy
// [[288]] 103 / 92 / 101 / 122 us, ML DEM 279 / 299 / 309 / 301 us, mix 126 / 125 / 125 /
// 138 us.
constexpr int kChunkMinBlocks = 5;

template <bool MLK>
__global__ void __launch_bounds__(kChunkWarps * 32, kChunkMinBlocks) chunk_kernel(const DevBatch b) {
  __shared__ ChunkArea areas[kChunkWarps];
  const int wib = threadIdx.x >> 5;
  const unsigned long long chunk = (unsigned long long)blockIdx.x * kChunkWarps + (unsigned)wib;
  if (chunk * (unsigned)b.chunk >= (unsigned long long)b.num_shots) return;
  // The first blocks of an SM find its L1 empty: one load per 128-byte line of the codes'
  // tables, and of the binomials of small sets, starts them on their way together, in
  // place of one miss after another along the search's chains.
  {
    const int stride = kChunkWarps * 32;
    for (int k = 0; k < b.num_codes && k < kWarmCodes; ++k) {
      const DevCode &cd = b.codes[k];
      const int lines = cd.g_gs ? (cd.g_words + 31) >> 5 : 0;
      for (int i = threadIdx.x; i < lines; i += stride) touch_line(cd.g_rows + 32 * i);
    }
    for (int i = threadIdx.x; i < kWarmTam * (kMaxW + 1) / 16; i += stride) touch_line(b.ncr + 16 * i);
  }
  const unsigned tag = *reinterpret_cast<volatile unsigned *>(b.epoch) + 1u;
  const unsigned long long t_enter = b.profile ? global_ns() : 0ull;
  ChunkStats st{0, 0, 0};
  classify_chunk<MLK, true>(b, (int)chunk, b.chunk, areas[wib].fast, &areas[wib], st, tag);
  if ((threadIdx.x & 31) == 0) {
    add_stats(b, st);
    if (b.profile) {
      const unsigned long long t = global_ns();
      unsigned long long *ends = ctr_ptr(b.counters, kCtrProfEnds);
      atomicMax(ends + kProfStart, ~t_enter);
      atomicMax(ends + kProfChunk, t);
      atomicAdd(ctr_ptr(b.counters, kCtrProfSums) + kProfChunk, t - t_enter);
      atomicAdd(ctr_ptr(b.counters, kCtrProfSums) + kProfSteps, 1ull);
    }
  }
}

}  // namespace grand
