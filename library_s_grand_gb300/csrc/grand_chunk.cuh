// grand_chunk.cuh -- the chunk step of a decoding launch (sm_103a): up to kMaxChunk launch slots
// by one warp, one lane per shot.
//
// classify_chunk
//   packs the shots' records with coalesced loads, forms each syndrome and settles the
//   common shots outright: an empty syndrome (grand_decoder.cu:1223-1241), and a first
//   threshold iteration with one active position whose column equals the syndrome
//   (weight-1 match, 1 candidate tested).  The others stay open: their syndromes wait in
//   the chunk's rows.
// write_chunk
//   writes the results of the chunk's settled shots, and appends those still open to
//   the slow queue of the decode kernel.
//
// The chunk kernel (grand_front.cuh) runs the guided search on the open shots in between;
// the decode kernel runs the two back to back for batches without a guided code.
#pragma once

#include "grand_kernels.cuh"

namespace grand {

// A syndrome: the second half is used by codes of more than 128 rows (wide).
struct Resid {
  uint4 a, b;
};
__device__ __forceinline__ void xor_into(uint4 &r, const uint4 w) {
  r.x ^= w.x;
  r.y ^= w.y;
  r.z ^= w.z;
  r.w ^= w.w;
}
__device__ __forceinline__ void xor_col(const uint32_t *cols, bool wide, unsigned c, Resid &r) {
  const uint4 *p = reinterpret_cast<const uint4 *>(cols) + (c << (wide ? 1 : 0));
  xor_into(r.a, __ldg(p));
  if (wide) xor_into(r.b, __ldg(p + 1));
}
// ---------------------------------------------------------------------------
// Chunks of up to kMaxChunk launch slots, one lane per shot.
// ---------------------------------------------------------------------------
// words of a chunk's separate logical entries (flat_ballots)
constexpr int kLogBallots = kMaxChunk * kFastLogWords + 8;

// A chunk in its warp's shared memory.  A shot's row holds its syndrome (words 0 .. 7),
// sketch (8), supplied weight (9) and logical words (10 .. 13) while it is open, and its
// result's 18 words once it is settled.
struct alignas(16) FastArea {
  uint32_t row[kMaxChunk][18];
  unsigned long long key[kMaxChunk];    // settled shots: the decoded columns (set_col), row[1] of them
  int shot[kMaxChunk], code[kMaxChunk];
  int at[kMaxChunk];                    // where its record starts in bits (-1: elsewhere, kKept:
                                        // in the record cache)
  uint8_t state[kMaxChunk];             // 0: open, 1: settled
  uint32_t bits[kFastBallots + 8];      // the run's records, entry after entry (flat_ballots)
};
constexpr int kKept = -2;
constexpr int kRowSketch = kFastWords, kRowWeight = kFastWords + 1, kRowLog = kFastWords + 2;
static_assert(kRowLog + kFastLogWords <= 18, "an open shot's words fit its row");
static_assert(sizeof(FastArea) + 4 * kLogBallots <= sizeof(WarpArea),
              "FastArea must fit the decode kernel's area");

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

// Column e (of w, in list order) of a column set: 10 bits each, the first on top.
__device__ __forceinline__ unsigned set_col(unsigned long long key, int w, int e) {
  return (unsigned)(key >> (10 * (w - 1 - e))) & 1023u;
}

// Word `lane` of the column set `key` (w columns).
__device__ __forceinline__ uint32_t set_word(unsigned long long key, int w) {
  const int lane = threadIdx.x & 31;
  uint32_t e = 0u;
#pragma unroll 1
  for (int k = 0; k < w; ++k) {
    const unsigned c = set_col(key, w, k);
    if ((int)(c >> 5) == lane) e |= 1u << (c & 31u);
  }
  return e;
}

// out[0 .. n) = the bits of word `lane` of a vector, one byte each.
__device__ __forceinline__ void bits_to_bytes(unsigned char *out, int n, uint32_t word) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int c0 = 0; c0 < n; c0 += 32) {
    const uint32_t w = __shfl_sync(kFull, word, c0 >> 5);
    if (c0 + lane < n) out[c0 + lane] = (unsigned char)((w >> lane) & 1u);
  }
}

// The record of a lane's shot (its bits from entry `at` of F.bits, its logical words from its row)
// into the record cache, for the per-shot path in place of a second read of the caller's.
// False: longer than a cache row.
static __device__ __noinline__ bool keep_record(const DevBatch &b, const HotCode &cd, const FastArea &F,
                                                int lane, int at, int slot) {
  const int nbits = cd.input_kind == kInErrors ? cd.m : cd.R, nwords = (nbits + 31) >> 5;
  const int nlw = cd.family == kDem ? cd.nlw : 0;
  if (nwords + nlw > kRecCacheWords) return false;
  uint32_t *cp = b.rec_cache + (size_t)slot * kRecCacheWords;
#pragma unroll 1
  for (int q = 0; q < nwords; ++q) cp[q] = flat_word(F.bits, at, q, nbits);
#pragma unroll 1
  for (int k = 0; k < nlw; ++k) cp[nwords + k] = F.row[lane][kRowLog + k];
  return true;
}

// Classifies the shots of launch slots size * chunk + [0, size), size <= kMaxChunk, into F.
// hot: the block's copies of the codes (nullptr: none); lbits: kLogBallots words of scratch.  Returns the mask of the lanes whose
// shots the guided search takes: open, with their syndrome, sketch, supplied weight and
// logical words in their row.
//
// The results of the settled shots are exactly those of the general path: the one position
// is the only candidate of the iteration (found at weight 1, rank 0; one candidate
// counted on either branch, hibrido 0 / -1), and its active set is the set of nonzero
// columns contained in the syndrome (flagged-check count = column weight, for
// 0/1 matrices regular or not), a solo column found by the syndrome's sketch.
template <bool MLK>
__device__ __forceinline__ unsigned classify_chunk(const DevBatch &b, const HotCode *hot, int chunk,
                                                   int size, FastArea &F, uint32_t *lbits,
                                                   ChunkStats &st) {
  const int lane = threadIdx.x & 31;
  const int first_slot = chunk * size;  // < num_shots (the sum with a lane need not be an int)
  const bool valid = lane < size && lane < b.num_shots - first_slot;
  const int slot = valid ? first_slot + lane : first_slot;
  const unsigned long long t_start = global_ns();
  unsigned long long tp = b.profile ? t_start : 0ull;
  const int shot = valid ? (b.shot_map ? b.shot_map[slot] : slot) : 0;
  const int ci = (valid && b.shot_code) ? b.shot_code[shot] : 0;
  const DevCode &full = b.codes[ci];
  const HotCode &cd = hot && ci < kHotCodes ? hot[ci] : static_cast<const HotCode &>(full);
  const bool errs = cd.input_kind == kInErrors;
  const bool dem = cd.family == kDem;
  const bool packed = cd.packed != 0;
  const int nw = cd.nw;
  const int nbits = errs ? cd.m : cd.R;       // entries of the record's leading bit vector
  const int nwords = (nbits + 31) >> 5;
  bool ok = valid && chunk_takes(cd);
  const long long rbase = valid ? (b.in_off ? b.in_off[shot] : (long long)shot * cd.rec_len) : 0;
  uint32_t *row = F.row[valid ? lane : 0];
  if (valid) {
    F.shot[lane] = shot;
    F.code[lane] = ci;
  }

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
      const int cnt = b.num_shots - first_slot < size ? b.num_shots - first_slot : size;
      lpad = flat_ballots(b.in_log + (long long)first_slot * cd.n_logicos, cnt * cd.n_logicos, lbits);
      __syncwarp();
    }
  }
  const uint32_t *cols = cd.g_gs ? cd.g_cols : full.cols;
  const uint32_t *hcol = cd.g_gs ? cd.g_hcol : full.hcol;
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
#pragma unroll
      for (int k = 0; k < kFastWords; ++k) row[k] = 0u;
      // the sketch: four rows at a time from the code's table, where it has one
#pragma unroll 1
      for (int k = 0; k < nw; ++k) {
        uint32_t w = word(k);
        row[k] = w;
        if (cd.g_gs) {
          const uint32_t *nib = cd.g_nib + 128 * k;
#pragma unroll
          for (int u = 0; u < 8; ++u) hs ^= __ldg(nib + 16 * u + ((w >> (4 * u)) & 15u));
        } else {
#pragma unroll 1
          for (; w; w &= w - 1u) hs ^= row_hash(k * 32 + __ffs((int)w) - 1);
        }
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
            else if (sep) w = flat_word(lbits, lpad + lane * cd.n_logicos, k, cd.n_logicos);
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
  // buffers): each run's entries through one pass of ballots.  Records the chunk does not
  // take are left out: with them a run could outgrow the ballot area.
  const int rlen = dem && !sep ? cd.R + cd.n_logicos : nbits;
  const bool mine = ok && !packed;
  const long long pend = __shfl_up_sync(kFull, rbase + rlen, 1);
  const bool pint = __shfl_up_sync(kFull, mine ? 1 : 0, 1) != 0;
  const unsigned members_all = __ballot_sync(kFull, mine);
  const unsigned all_starts = __ballot_sync(kFull, mine && (lane == 0 || !pint || pend != rbase));
  const bool one_run = (all_starts & (all_starts - 1u)) == 0u;
  int at = 0;  // where this lane's record starts in the ballots
  bool kept = false;
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
    if (in_run && ok) {
      take(at, rw);
      // (the next run's bits take the place of these; a guided search seldom leaves a shot)
      if (!one_run && !rw && !cd.g_gs && b.rec_cache)
        kept = keep_record(b, cd, F, lane, at, slot);
    }
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
    const uint32_t mask = cd.g_gs ? cd.g_tab_mask : full.solo_mask;
    uint32_t i = hs & mask;
#pragma unroll 1
    for (uint32_t probe = 0; probe <= mask && !found; ++probe) {
      uint2 e;
      if (cd.g_gs) e = __ldg(reinterpret_cast<const uint2 *>(cd.g_tab) + i);
      else e = make_uint2(__ldg(full.solo_keys + i), (unsigned)__ldg(full.solo_cols + i) | kSoloFlag);
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
    }
  }
  if (valid) {
    F.state[lane] = done ? 1 : 0;
    F.key[lane] = found ? (unsigned long long)pos : 0ull;
    // (one run: its bits stay; a later run takes an earlier one's place)
    F.at[lane] = ok && !packed && one_run ? at : (kept ? kKept : -1);
  }
  __syncwarp();
  prof_lap(b, kProfChunkWrite, tp);
  return __ballot_sync(kFull, ok && !done && cd.g_gs);
}

// The chunk's results, and its open shots into the slow queue with tag (the launch
// epoch + 1).
//
// kCtrChunks counts the chunks done (high half) and the queue entries reserved (low
// half) in one word, so that a warp that sees every chunk done sees every
// reservation too, with no fence in between.
__device__ __forceinline__ void write_chunk(const DevBatch &b, const HotCode *hot, int chunk, int size,
                                            const FastArea &F, unsigned tag) {
  const int lane = threadIdx.x & 31;
  const int first_slot = chunk * size;
  const bool valid = lane < size && lane < b.num_shots - first_slot;
  const int slot = valid ? first_slot + lane : first_slot;
  const bool open = valid && F.state[valid ? lane : 0] == 0;
  const unsigned settled = __ballot_sync(kFull, valid && !open);
  const unsigned slow = __ballot_sync(kFull, open);
  // one coalesced pass over the rows: word i belongs to lane i / 18's shot
#pragma unroll 1
  for (int i = lane; i < size * 18; i += 32) {
    const int j = (i * 3641) >> 16;  // i / 18 for i < 18 * kMaxChunk
    if ((settled >> j) & 1u)
      reinterpret_cast<uint32_t *>(b.results + F.shot[j])[i - 18 * j] = F.row[j][i - 18 * j];
  }
  if (b.deferred && valid && !open) b.deferred[F.shot[lane]] = 0;
  if (b.dec_err || b.dec_log) {
#pragma unroll 1
    for (unsigned mm = settled; mm; mm &= mm - 1u) {
      const int j = __ffs((int)mm) - 1;
      const int sj = F.shot[j], w = (int)F.row[j][1];
      const unsigned long long key = F.key[j];
      const HotCode &cd = b.codes[F.code[j]];
      if (b.dec_err && cd.m <= kGuidedMaxCols) {
        bits_to_bytes(b.dec_err + (size_t)sj * cd.m, cd.m, set_word(key, w));
      } else if (b.dec_err) {  // one column at most: only the solo test settles such a code's shots
#pragma unroll 1
        for (int c = lane; c < cd.m; c += 32)
          b.dec_err[(size_t)sj * cd.m + c] = w && c == (int)key ? 1 : 0;
      }
      if (b.dec_log && cd.family == kDem) {
        uint32_t le = 0u;
#pragma unroll 1
        for (int k = 0; k < w && lane < cd.nlw; ++k)
          le ^= __ldg(cd.lcols + (w == 1 ? (unsigned)key : set_col(key, w, k)) * (unsigned)cd.nlw +
                      (unsigned)lane);
        bits_to_bytes(b.dec_log + (size_t)sj * cd.n_logicos, cd.n_logicos, le);
      }
    }
  }
  if (b.guided == kGuidedAll) {
    if (slow && lane == 0) atomicOr(b.status, kStatusWaitLimit);  // never: see guided_closed
    return;
  }
  unsigned long long base = 0;
  if (lane == 0)
    base = atomicAdd(ctr_ptr(b.counters, kCtrChunks), (1ull << 32) + (unsigned long long)__popc(slow));
  if (slow) {
    base = __shfl_sync(kFull, base, 0) & 0xffffffffull;
    if (open) {
      const int ci = F.code[lane], at = F.at[lane];
      const HotCode &cd = hot && ci < kHotCodes ? hot[ci] : static_cast<const HotCode &>(b.codes[ci]);
      const bool cache = at == kKept || (b.rec_cache && at >= 0 && keep_record(b, cd, F, lane, at, slot));
      // The record's bits before the entry, for a ticket holder that reads the entry at once: without
      // this some read an earlier round's record (6 of 10^6 shots, 5000 a batch, all heavy).
      // (After a chunk kernel they are read by the next launch.)
      if (cache && !b.guided) __threadfence();
      // the entry carries this launch's tag: a ticket holder that reads it knows it
      // is not a leftover of an earlier launch
      *reinterpret_cast<volatile unsigned long long *>(b.queue + base + __popc(slow & ((1u << lane) - 1u))) =
          ((unsigned long long)tag << 32) | (unsigned)slot | (cache ? 0x80000000u : 0u);
    }
  }
  __syncwarp();
}

}  // namespace grand
