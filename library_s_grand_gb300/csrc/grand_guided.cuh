// grand_guided.cuh -- the guided search, four shots to a warp (sm_103a).
//
// A set S of active columns matches when the XOR of its columns is the syndrome
// s.  Take any set row r of s: an odd number of S's columns hold r, so at least
// one of the few active columns that meet r is in S; remove it, and the same holds
// for the residual syndrome and the rest of S.  So every match of weight w is reached
// by choosing w - 1 columns, each among the active columns of the lowest set row
// of the residual so far, and looking the last column up by the residual's sketch
// -- at most deg^(w-1) steps (216 for a weight-4 pattern of a code whose rows
// meet 6 columns) where enumerating the (w-1)-prefixes takes C(tam, w-1) (317750 at
// tam = 126).  A residual of zero with columns still to choose has no row to
// follow: there every active column is tried.  A residual with more set rows than
// the columns left can hold (max column weight each) is dropped.
//
// All matches of a weight are found, so the one upstream's enumeration reaches
// first is the least of them: for a first-hit search the lexicographically
// smallest column set (the active list is ascending, so index order is column
// order), for ML the least FP32 cost (LLRs summed in the list's order, ascending by
// LLR then column) with ties to the smaller index set.  Its rank in the enumeration,
// and with it the number of candidates upstream reports, follow from its positions.
//
// Levels.  The partial sets of one size, of all the warp's shots, lie side by side in
// shared memory ("items": the item extended and the column added, the residual's sketch
// and lowest row, the shot).  Level d extends the items of d - 1 columns by one: the
// warp's lanes take (item, neighbour) pairs, so a level of n items is n * deg / 32
// steps whatever the shape of the trees; each new set probes the sketch filter for its
// last column (weight d + 1) and, while larger weights remain, is kept for the next
// level.  Shots whose levels together outgrow the items are searched again one by one;
// one that outgrows them alone takes the general path, and so does one with a level of more
// than kLevelPairs (item, neighbour) pairs, where a decode kernel follows: its warps share
// such a search, which this one would walk while the rest of the GPU waits for it.
//
// The flagged-check counts (upstream grand_decoder.cu:67-81, 406-416) are formed
// from the rows: a lane holds a mask word of the columns, the rows of H selected by
// the syndrome are added into 3-bit counters kept as bit slices, and a column is
// active in iteration i when at most i of its rows are missing from the syndrome
// (its count, with the irregular offset, reaches max_soma - i).
//
// What bounds it: the instruction chain (some 11 cycles an instruction per warp, L1 round
// trips among them) and the instruction caches.  Most of a shot's instructions are
// uniform -- planning, loop control, reductions -- so eight lanes take a shot and a
// warp takes four, in step; the code is kept small: loops stay rolled, column widths
// are a run-time choice and the rare parts are out of line.  Headline batch 28.9 us, mix of
// 100000 shots 60, noisy [[288]] 51, random detectors of the 720-mechanism DEM 24.5; with
// a shot per warp 43.7, 112, 88 and 34, in the decode kernel alone 82, 237, 939 and 568.
#pragma once

#include "grand_chunk.cuh"

namespace grand {

// One shot of the warp: its syndrome, the active columns of its iterations, and what the
// lanes that extend its sets read of its code.
struct alignas(16) GuidedGroup {
  uint32_t sw[8];                    // the syndrome, zero past nw
  uint32_t am[kMaxIters][32];        // the iterations' active columns
  const uint32_t *cols, *hcol, *filt, *tab;
  const uint16_t *adj;
  const float *llr;                  // nullptr: first-hit search
  uint32_t tab_mask;
  int deg, m;
  int limit;                         // most set rows a residual of this level may have
  int wide;                          // more than 128 rows: columns of eight words
};
// An item: x: the residual's sketch; y: the item it extends (10 bits), the column added
// (10), the residual's lowest row (10, kNoRow: zero) and the group (2).
struct alignas(16) GuidedArea {
  uint2 item[kGuidedItems];
  uint32_t queue[64];  // children waiting: item << 10 | column
  GuidedGroup group[32 / kGuidedLanes];
};
constexpr unsigned kNoRow = 1023u;
// The syndromes' set rows, ascending, padded with R: a byte each, where the items go later.
constexpr int kRowList = (kGuidedMaxRows + 4 + 7) & ~7;
static_assert(32 / kGuidedLanes * kRowList <= (int)sizeof(uint2) * kGuidedItems, "row lists fit the items");
static_assert(kGuidedItems <= 1024 && kGuidedMaxCols <= 1024 && kGuidedMaxRows < (int)kNoRow &&
                  32 / kGuidedLanes <= 4,
              "an item's fields have 10 bits each, its group 2");

// The columns of a partial set, 16 bits each from the lowest up (the rest kNoCol).
struct Path {
  uint32_t lo, hi;
};
__device__ __forceinline__ void push_col(Path &p, unsigned c) {
  p.hi = (p.hi << 16) | (p.lo >> 16);
  p.lo = (p.lo << 16) | c;
}
__device__ __forceinline__ unsigned pop_col(Path &p) {
  const unsigned c = p.lo & 0xffffu;
  p.lo = (p.lo >> 16) | (p.hi << 16);
  p.hi >>= 16;
  return c;
}
__device__ __forceinline__ bool in_path(const Path &p, unsigned c) {
  return c == (p.lo & 0xffffu) || c == p.lo >> 16 || c == (p.hi & 0xffffu) || c == p.hi >> 16;
}
// The syndrome XOR the d columns of p and column c.
__device__ __forceinline__ Resid residual(const uint32_t *sw, const uint32_t *cols, bool wide, Path p,
                                          int d, unsigned c) {
  Resid r;
  r.a = *reinterpret_cast<const uint4 *>(sw);
  r.b = *(reinterpret_cast<const uint4 *>(sw) + 1);
  xor_col(cols, wide, c, r);
#pragma unroll 1
  for (; d > 0; --d) xor_col(cols, wide, pop_col(p), r);
  return r;
}

__device__ __forceinline__ int ones_of(const Resid &r) {
  return __popc(r.a.x) + __popc(r.a.y) + __popc(r.a.z) + __popc(r.a.w) + __popc(r.b.x) +
         __popc(r.b.y) + __popc(r.b.z) + __popc(r.b.w);
}
// Lowest set row of a residual (kNoRow: zero).
__device__ __forceinline__ unsigned lowest_row(const Resid &r) {
  uint32_t w = r.b.w;
  unsigned at = 224u;
  if (r.b.z) w = r.b.z, at = 192u;
  if (r.b.y) w = r.b.y, at = 160u;
  if (r.b.x) w = r.b.x, at = 128u;
  if (r.a.w) w = r.a.w, at = 96u;
  if (r.a.z) w = r.a.z, at = 64u;
  if (r.a.y) w = r.a.y, at = 32u;
  if (r.a.x) w = r.a.x, at = 0u;
  return w ? at + (unsigned)__ffs((int)w) - 1u : kNoRow;
}

// The best match a lane has seen of the weight being searched: first-hit the set
// as ascending 10-bit columns (key), ML the cost key with the set in list order.
struct GuidedBest {
  unsigned long long key;
  uint32_t cost;
};

// ML: is index set a before b in the enumeration (both in list order)?
__device__ __forceinline__ bool ml_set_before(const float *llr, unsigned long long a,
                                              unsigned long long b, int w) {
#pragma unroll 1
  for (int e = 0; e < w; ++e) {
    const unsigned x = set_col(a, w, e), y = set_col(b, w, e);
    if (x == y) continue;
    const float lx = __ldg(llr + x), ly = __ldg(llr + y);
    return lx < ly || (lx == ly && x < y);
  }
  return false;
}

// The set {the d columns of p, c, j}, when it XORs to the syndrome, into the lane's
// best after it.  Rare, so out of line (everything by value: what it is called with
// stays in registers).  c == kNoCol: the set {j}.
template <bool MLK>
__device__ __noinline__ GuidedBest guided_match(const uint32_t *sw, const uint32_t *cols, bool wide,
                                                const float *llr, Path p, int d, unsigned c,
                                                unsigned j, GuidedBest best) {
  Resid r = residual(sw, cols, wide, p, d, j);
  if (c != kNoCol) xor_col(cols, wide, c, r);
  if (ones_of(r)) return best;  // equal sketches, different columns
  const bool ml = MLK && llr != nullptr;
  // the columns in list order, by insertion: 10 bits each, the first on top
  const int w = d + (c != kNoCol ? 2 : 1);
  unsigned long long key = 0ull;
#pragma unroll 1
  for (int e = 0; e < w; ++e) {
    const unsigned x = e < d ? pop_col(p) : (e == w - 1 ? j : c);
    const float lx = ml ? __ldg(llr + x) : 0.0f;
    int at = e;  // columns after x among the e placed
#pragma unroll 1
    for (int f = 0; f < e; ++f) {
      const unsigned y = (unsigned)(key >> (10 * f)) & 1023u;  // from the last one up
      const float ly = ml ? __ldg(llr + y) : 0.0f;
      if (ly < lx || (ly == lx && y < x)) {
        at = f;
        break;
      }
    }
    const unsigned long long tail = key & ((1ull << (10 * at)) - 1ull);
    key = ((((key >> (10 * at)) << 10) | x) << (10 * at)) | tail;
  }
  if (!ml) {
    if (key < best.key) best.key = key;
    return best;
  }
  float cost = 0.0f;
#pragma unroll 1
  for (int e = 0; e < w; ++e) cost = __fadd_rn(cost, __ldg(llr + set_col(key, w, e)));
  const uint32_t o = cost_key(cost);
  if (o < best.cost || (o == best.cost && ml_set_before(llr, key, best.key, w))) {
    best.cost = o;
    best.key = key;
  }
  return best;
}

// The active columns outside the set whose sketch is h, each tested as the last
// column of the set {the d columns of p, c}.
template <bool MLK>
__device__ __forceinline__ void guided_probe(const GuidedGroup &S, const uint32_t *am, const Path &p,
                                             int d, unsigned c, uint32_t h, GuidedBest &best) {
  const uint32_t f = h >> (32 - kGuidedF);
  if (!((__ldg(S.filt + (f >> 5)) >> (f & 31u)) & 1u)) return;
  const uint32_t mask = S.tab_mask;
  uint32_t i = h & mask;
#pragma unroll 1
  for (uint32_t guard = 0; guard <= mask; ++guard) {
    const uint2 e = __ldg(reinterpret_cast<const uint2 *>(S.tab) + i);
    const unsigned j = e.y & 0xffffu;
    if (j == kNoCol) return;
    if (e.x == h && j != c && !in_path(p, j) && ((am[j >> 5] >> (j & 31u)) & 1u))
      best = guided_match<MLK>(S.sw, S.cols, S.wide != 0, MLK ? S.llr : nullptr, p, d, c, j, best);
    i = (i + 1u) & mask;
  }
}

// What the search found for a group's shot.
struct GuidedWinner {
  int w;                    // 0: nothing
  unsigned long long key;   // its columns, in list order
  uint32_t cost;            // ML cost key
  int w_done;               // ML: last weight searched (the bound may stop it early)
};

// Four rows added to the counters of each bit position (mod 8), by full adders.
__device__ __forceinline__ uint32_t majority(uint32_t a, uint32_t b, uint32_t c) {
  return (a & b) | (a & c) | (b & c);
}
__device__ __forceinline__ void add_rows(uint32_t x0, uint32_t x1, uint32_t x2, uint32_t x3,
                                         uint32_t &c0, uint32_t &c1, uint32_t &c2) {
  const uint32_t s = x0 ^ x1 ^ x2, m = majority(x0, x1, x2);
  const uint32_t n = majority(c0, s, x3);
  c0 ^= s ^ x3;
  c2 ^= majority(c1, m, n);
  c1 ^= m ^ n;
}

// Are the bits of delta (word `lane` of the difference of two errors with one syndrome)
// in the row space of the other matrix (grand_decoder.cu:456-474)?  The XOR of its reduced
// rows pivoted on delta's bits equals delta exactly then.
static __device__ __noinline__ bool in_row_space(const DevCode &cd, uint32_t delta) {
  const int lane = threadIdx.x & 31;
  const int mw = cd.mw;
  uint32_t acc = 0u;
#pragma unroll 1
  for (unsigned words = __ballot_sync(kFull, delta != 0u); words; words &= words - 1u) {
    const int q = __ffs((int)words) - 1;
    const uint32_t word = __shfl_sync(kFull, delta, q);
    const int r = ((word >> lane) & 1u) ? __ldg(cd.pivrow + q * 32 + lane) : -1;
    unsigned piv = __ballot_sync(kFull, r >= 0);
#pragma unroll 1
    while (piv) {
      uint32_t x[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {  // four rows in flight
        const int rb = __shfl_sync(kFull, r, piv ? __ffs((int)piv) - 1 : 0);
        x[u] = piv && lane < mw ? __ldg(cd.rref + rb * mw + lane) : 0u;
        piv &= piv - 1u;
      }
      acc ^= x[0] ^ x[1] ^ x[2] ^ x[3];
    }
  }
  return __all_sync(kFull, acc == delta);
}

// Word `lane` of a supplied error (CSS): from its chunk's ballots (at >= 0) or from the
// record itself.
static __device__ __noinline__ uint32_t error_word(const DevBatch &b, const HotCode &cd, const FastArea &F,
                                                   int at, int shot) {
  const int lane = threadIdx.x & 31;
  const int rem = cd.m - 32 * lane;
  if (at >= 0) return rem > 0 ? flat_word(F.bits, at, lane, cd.m) : 0u;
  const int *rec = b.in + (b.in_off ? b.in_off[shot] : (long long)shot * cd.rec_len);
  if (cd.packed)
    return rem > 0 ? (unsigned)__ldcg(rec + lane) & (rem < 32 ? (1u << rem) - 1u : kFull) : 0u;
  uint32_t mine = 0u;
#pragma unroll 1
  for (int q = 0; 32 * q < cd.m; ++q) {
    const uint32_t w = __ballot_sync(kFull, 32 * q + lane < cd.m && __ldcg(rec + 32 * q + lane) != 0);
    if (q == lane) mine = w;
  }
  return mine;
}

// The groups whose items among lo .. hi - 1 make more than kLevelPairs pairs, as a mask (rare).
static __device__ __noinline__ int long_groups(const GuidedArea &A, int lo, int hi, int deg) {
  const int lane = threadIdx.x & 31;
  unsigned long long n = 0ull;  // items per group, 16 bits each
#pragma unroll 1
  for (int i = lo + lane; i < hi; i += 32) n += 1ull << (16 * (A.item[i].y >> 30));
#pragma unroll 1
  for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(kFull, n, o);
  int mask = 0;
#pragma unroll 1
  for (int k = 0; k < 32 / kGuidedLanes; ++k)
    if ((int)((n >> (16 * k)) & 0xffffu) * deg > kLevelPairs) mask |= 1 << k;
  return mask;
}

// cnt (1 .. 4) open shots of the block: the threshold iterations in upstream's order
// (grand_decoder.cu:1284-1343) until one has a match, and the shot's result into its row.
// An entry is (warp of the block << 8) | lane of its chunk.  Returns the mask of the shots
// finished (bit k: entry k; none of them when the levels do not fit), in bits 8 .. those past
// the light budget, and in bits 16 .. those that a level's length leaves to the decode kernel
// (then none is finished).
//
// Eight lanes (a group) count, plan and report for one shot; the sets are extended by
// all lanes for all of them.  The groups run in step: every loop goes on while some group
// needs it, and a collective of the warp serves all of them.
template <bool MLK>
__device__ __noinline__ int guided_pass(const DevBatch &b, const HotCode *hot, GuidedArea &A,
                                        FastArea *areas, size_t area_step, const uint16_t *list,
                                        int cnt) {
  constexpr int G = kGuidedLanes;
  constexpr unsigned kGroup = (1u << G) - 1u;
  const int lane = threadIdx.x & 31;
  const int g = lane / G, gl = lane & (G - 1), gb = g * G;
  GuidedGroup &S = A.group[g];
  uint2 *item = A.item;
  uint8_t *row_list = reinterpret_cast<uint8_t *>(A.item) + g * kRowList;
  const unsigned long long t_start = global_ns();
  unsigned long long tp = b.profile ? t_start : 0ull;
  bool live = g < cnt;
  const int entry = live ? (int)list[g] : 0;
  FastArea &F = *reinterpret_cast<FastArea *>(reinterpret_cast<char *>(areas) + (entry >> 8) * area_step);
  const int j = entry & 255;
  uint32_t *row = F.row[j];
  const int ci = F.code[j];
  const DevCode &full = b.codes[ci];
  const HotCode &cd = hot && ci < kHotCodes ? hot[ci] : static_cast<const HotCode &>(full);
  const bool ml = MLK && cd.variant == kMl;
  const bool prob = cd.variant == kProb;
  const int mw = cd.mw, max_cw = cd.g_max_cw;
  const float *llr = ml ? cd.llr : nullptr;
  // (a group without a shot reads nothing of entry 0's, which its warp may be writing)
  const uint32_t hs = live ? row[kRowSketch] : 0u;
  if (gl == 0) {
    S.cols = cd.g_cols;
    S.hcol = cd.g_hcol;
    S.filt = cd.g_filt;
    S.tab = cd.g_tab;
    S.adj = cd.g_adj;
    S.llr = llr;
    S.tab_mask = cd.g_tab_mask;
    S.deg = cd.g_deg;
    S.m = cd.m;
    S.wide = cd.g_gs == 8 ? 1 : 0;
  }
  // the largest row degree of the warp's codes: the pairs an item is given
  int deg = cd.g_deg;
  unsigned long long magic = cd.g_magic;
#pragma unroll 1
  for (int o = G; o < 32; o <<= 1) {
    const int d2 = __shfl_xor_sync(kFull, deg, o);
    const unsigned long long m2 = __shfl_xor_sync(kFull, magic, o);
    if (d2 > deg) {
      deg = d2;
      magic = m2;
    }
  }

  // ---- the syndrome and its rows: lane gl the rows of word gl ----------------------
  int ones;
  {
    uint32_t word = gl < kFastWords && live ? row[gl] : 0u;
    if (gl < kFastWords) S.sw[gl] = word;
    int sum = __popc(word);
    const int mine = sum;
#pragma unroll 1
    for (int o = 1; o < kFastWords; o <<= 1) {
      const int u = __shfl_sync(kFull, sum, lane - o);
      if (gl >= o) sum += u;
    }
    ones = __shfl_sync(kFull, sum, gb + kFastWords - 1);
    int n = sum - mine;
#pragma unroll 1
    for (; word; word &= word - 1u) row_list[n++] = (uint8_t)(32 * gl + __ffs((int)word) - 1);
    if (gl < 4) row_list[ones + gl] = (uint8_t)cd.R;  // the row of zeros behind the table's
  }
  __syncwarp();
  const unsigned row0 = row_list[0];

  // ---- counts, bit-sliced: lane gl the columns of mask words gl, gl + G, .. ----------
  const int L = cd.max_soma < kMaxIters ? cd.max_soma : kMaxIters;
  int t01 = 0, t2 = 0;  // active columns of the iterations (the first two packed)
#pragma unroll 1
  for (int q = gl; __any_sync(kFull, live && q < mw); q += G) {
    if (live && q < mw) {
      const uint32_t *rows = cd.g_rows + q;
      uint32_t c0 = 0u, c1 = 0u, c2 = 0u;
#pragma unroll 1
      for (int i = 0; i < ones; i += 4) {
        const uchar4 r = *reinterpret_cast<const uchar4 *>(row_list + i);
        const uint32_t x0 = __ldg(rows + (int)r.x * mw), x1 = __ldg(rows + (int)r.y * mw),
                       x2 = __ldg(rows + (int)r.z * mw), x3 = __ldg(rows + (int)r.w * mw);
        add_rows(x0, x1, x2, x3, c0, c1, c2);
      }
      const uint32_t w0 = __ldg(cd.g_cw + q), w1 = __ldg(cd.g_cw + mw + q), w2 = __ldg(cd.g_cw + 2 * mw + q);
      // missing = weight - count, bit by bit; zero columns are never active
      const uint32_t nz = w0 | w1 | w2;
      const uint32_t m0 = w0 ^ c0, b0 = ~w0 & c0;
      const uint32_t m1 = w1 ^ c1 ^ b0, b1 = (~w1 & c1) | (~(w1 ^ c1) & b0);
      const uint32_t m2 = w2 ^ c2 ^ b1;
      const uint32_t a0 = nz & ~(m0 | m1 | m2), a1 = nz & ~(m1 | m2), a2 = nz & ~(m2 | (m1 & m0));
      S.am[0][q] = a0;
      S.am[1][q] = a1;
      S.am[2][q] = a2;
      t01 += __popc(a0) | (__popc(a1) << 16);
      t2 += __popc(a2);
    }
  }
#pragma unroll 1
  for (int o = 1; o < G; o <<= 1) {
    t01 += __shfl_xor_sync(kFull, t01, o);
    t2 += __shfl_xor_sync(kFull, t2, o);
  }
  __syncwarp();
  const unsigned long long t_counts = global_ns();
  tp = prof_lap(b, kProfShotCounts, tp);

  // ---- the iterations --------------------------------------------------------------
  GuidedWinner wn;
  wn.w = 0;
  wn.key = kNone;
  int tam = 0, tam_old = 0, passes = 0, hib = -2, heavy = 0, found = 0;
  unsigned long long tested = 0;
#pragma unroll 1
  for (int i = 0; i < kMaxIters; ++i) {
    bool on = live && !found && i < L;
    if (!__any_sync(kFull, on)) break;
    const int n_act = i == 0 ? t01 & 0xffff : (i == 1 ? t01 >> 16 : t2);
    uint32_t *am = S.am[i];
    if (on) {
      passes = i + 1;
      tam = n_act;
      if (cd.family == kDem) {  // grand_decoder.cu:1550-1554
        if (tam > cd.cap) tam = tam_old;
        else tam_old = tam;
      }
    }
    const bool gpu = (tam > cd.thr && tam <= cd.cap && cd.mode == 1) || cd.mode == 0;
    const bool cpu = !gpu && ((tam <= cd.thr && cd.mode == 1) || cd.mode == -1);
    on = on && tam > 0 && (gpu || cpu);
    if (__any_sync(kFull, on && tam < n_act)) {
      // the first tam columns of the larger set (the cap rule)
      int left = on ? tam : n_act;
#pragma unroll 1
      for (int q0 = 0; __any_sync(kFull, q0 < mw); q0 += G) {
        const int q = q0 + gl;
        uint32_t word = q < mw ? am[q] : 0u;
        int sum = __popc(word);
        const int mine = sum;
#pragma unroll 1
        for (int o = 1; o < G; o <<= 1) {
          const int u = __shfl_sync(kFull, sum, lane - o);
          if (gl >= o) sum += u;
        }
        int keep = left - (sum - mine);
        if (keep < mine && q < mw) {
          uint32_t cut = 0u;
#pragma unroll 1
          for (; keep > 0; --keep) {
            cut |= word & (0u - word);
            word &= word - 1u;
          }
          am[q] = cut;
        }
        left -= __shfl_sync(kFull, sum, gb + G - 1);
      }
      __syncwarp();
    }
    // candidate counts: lane k of the group holds those of weights 1 .. k
    const unsigned long long upto = gl < 8 ? __ldg(b.upto + 8 * tam + gl) : 0ull;

    // the weights searched (bit w), in one ascending run or weight 6 (run) before the others
    unsigned ws = 0u, run = 0u;
    const int *order = full.mask_order[0];
    int wmax = cd.Wc < tam ? cd.Wc : tam;
    if (on && prob) {
      int mi = cd.n_masks - 1;  // grand_decoder.cu:754-762
#pragma unroll 1
      for (int q = 0; q < cd.n_masks; ++q)
        if (tam <= full.mask_tam_upper[q]) {
          mi = q;
          break;
        }
      order = full.mask_order[mi];
#pragma unroll 1
      for (int k = 0; k < cd.num_phases; ++k) {
        const int pid = order[k];
        if (pid == 0) ws |= (2u << (tam < 5 ? tam : 5)) - 2u;
        if (pid == 1 && tam >= 6) {
          if (!ws) run = 64u;
          ws |= 64u;
        }
      }
      if (!run) run = ws;
    } else if (on) {
      run = ws = (2u << wmax) - 2u;
    }
    unsigned rest = ws & ~run;

    // ---- the search ------------------------------------------------------------------
#pragma unroll 1
    while (__any_sync(kFull, run != 0u)) {
      const int w_first = run ? __ffs((int)run) - 1 : 1;
      int w_last = run ? 31 - __clz((int)run) : 0;
      if (run) {
        wn.w = 0;
        wn.cost = 0xffffffffu;
        wn.w_done = w_last;
      }
      // columns of odd weight only: the weight of a match and the syndrome's are alike
      // (ML goes on to the last weight for its bound)
      const bool odd = cd.g_odd != 0;
      if (odd && !ml && ((w_last ^ ones) & 1)) --w_last;
      bool go = run != 0u && w_last >= w_first && ones <= max_cw * w_last;
      // the roots: the empty sets of the groups that search
      unsigned roots = __ballot_sync(kFull, go && gl == 0);
      int lo = 0, hi = __popc(roots);
      if (go && gl == 0)
        item[__popc(roots & ((1u << lane) - 1u))] = make_uint2(hs, ((unsigned)g << 30) | row0);
      __syncwarp();
      float psum = 0.0f;                // ML: sum of the pw smallest LLRs of the active set,
      unsigned long long plast = 0ull;  //   {LLR key, column} of the last of them, plus one
      int pw = 0;
      float floor = 0.0f;  // ML: w times the code's least LLR, added up as the prefix sums are
#pragma unroll 1
      for (int w = 1; __any_sync(kFull, go && w <= w_last); ++w) {
        bool act = go && w <= w_last;
        // The bound: the search stops where the sum of the w smallest LLRs reaches the best
        // cost.  That sum is no less than floor (FP32 addition is monotonic), which mostly
        // settles it; only otherwise is it formed (65536 shots of the 720-mechanism DEM,
        // drawing them included: 134 us, 139 with the sum formed for every weight).
        if (MLK && ml) {
          floor = __fadd_rn(floor, cd.llr_min);
          if (act && wn.w && floor >= key_cost(wn.cost)) {
            wn.w_done = w - 1;
            go = act = false;
          }
        }
        if (MLK && __any_sync(kFull, act && ml && wn.w)) {
          // upstream's prefix sums: the w smallest LLRs, added in ascending order
#pragma unroll 1
          for (;;) {
            const bool want = act && ml && wn.w && pw < w;
            if (!__any_sync(kFull, want)) break;
            unsigned long long next = kNone;
            if (want) {
#pragma unroll 1
              for (int q = gl; q < mw; q += G)
#pragma unroll 1
                for (uint32_t word = am[q]; word; word &= word - 1u) {
                  const int c = 32 * q + __ffs((int)word) - 1;
                  const uint32_t u = __float_as_uint(__ldg(llr + c));
                  const uint32_t k = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
                  const unsigned long long x = ((unsigned long long)k << 32) | (unsigned)c;
                  if (x >= plast && x < next) next = x;
                }
            }
#pragma unroll 1
            for (int o = 1; o < G; o <<= 1) {
              const unsigned long long u = __shfl_xor_sync(kFull, next, o);
              next = u < next ? u : next;
            }
            if (next != kNone) {
              const uint32_t k = (uint32_t)(next >> 32);
              psum = __fadd_rn(psum, __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k));
              plast = next + 1ull;
            }
            if (want) ++pw;
          }
          if (act && ml && wn.w && psum >= key_cost(wn.cost)) {
            wn.w_done = w - 1;
            go = act = false;
          }
        }
        const int d = w - 1;  // columns of the sets formed
        // bit gb of a mask: the group's
        const unsigned acts = __ballot_sync(kFull, act);
        const unsigned probes = __ballot_sync(kFull, act && w >= w_first && !(odd && ((w ^ ones) & 1)));
        const unsigned pushes = __ballot_sync(kFull, act && w < w_last);
        if (d == 0) {
          // weight 1 ends here unless a root's sketch passes its filter
          const uint32_t f = hs >> (32 - kGuidedF);
          const bool pass = gl == 0 && ((probes >> gb) & 1u) &&
                            ((__ldg(cd.g_filt + (f >> 5)) >> (f & 31u)) & 1u);
          if (!__any_sync(kFull, pass)) continue;
        }
        if (gl == 0) S.limit = max_cw * (w_last - d);
        __syncwarp();
        unsigned long long bkey = kNone;  // the group's best of this weight
        uint32_t bcost = 0xffffffffu;
        const Path none{0xffffffffu, 0xffffffffu};
        const int pairs = d == 0 ? hi : (hi - lo) * deg;
        if (pairs > kLevelPairs && b.guided != kGuidedAll) {
          const int left = long_groups(A, lo, hi, deg);
          if (left) return left << 16;
        }
        int top = hi, queued = 0;
        bool zeros = false, drained = false;
        int zi = -1;  // an item of residual zero being extended by every active column
        uint32_t zbits = 0u;
        // The children are found in steps of 32 (item, neighbour) pairs (weight 1: the
        // roots), then, for each item without a row to follow, in steps over its group's active
        // columns, a lane those of its word.  Most pairs' columns are not active (nearly
        // all in a DEM, whose rows meet dozens), so the ones that are queue up, and are
        // taken 32 at a time (sampled ML DEM, with the row lists moved into the items'
        // place: 152 -> 142 us; the BB batches within 2 %).
#pragma unroll 1
        for (int p0 = 0; !drained; p0 += 32) {
          unsigned entry = 0u;  // item << 10 | column
          bool found_one = false;
          if (p0 < pairs) {
            const int p = p0 + lane;
            if (d == 0) {
              entry = (unsigned)lane << 10;
              found_one = lane < hi;
            } else if (p < pairs) {
              const int n = (int)(((unsigned long long)(unsigned)p * magic) >> 32);
              const int k = p - n * deg;
              const uint32_t y = item[lo + n].y;
              const GuidedGroup &T = A.group[y >> 30];
              const unsigned r = y & 1023u;
              if (r == kNoRow) {
                zeros = true;
              } else if (k < T.deg && ((acts >> (G * (y >> 30))) & 1u)) {
                const unsigned c = __ldg(T.adj + r * (unsigned)T.deg + (unsigned)k);
                entry = ((unsigned)(lo + n) << 10) | c;
                found_one = c != kNoCol && ((T.am[i][(c >> 5) & 31u] >> (c & 31u)) & 1u);
              }
            }
            if (p0 + 32 >= pairs) drained = !__any_sync(kFull, zeros);  // (ML, or weights out of order)
          } else {
            if (!__any_sync(kFull, zbits != 0u)) {
              zi = zi < 0 ? lo : zi + 1;
              while (zi < hi && !((item[zi].y & 1023u) == kNoRow && ((acts >> (G * (item[zi].y >> 30))) & 1u)))
                ++zi;
              drained = zi >= hi;
              if (!drained) {
                const GuidedGroup &T = A.group[item[zi].y >> 30];
                zbits = 32 * lane < T.m ? T.am[i][lane] : 0u;
              }
            }
            if (zbits) {
              entry = ((unsigned)zi << 10) | (unsigned)(32 * lane + __ffs((int)zbits) - 1);
              found_one = true;
              zbits &= zbits - 1u;
            }
          }
          const unsigned fresh = __ballot_sync(kFull, found_one);
          if (found_one) A.queue[queued + __popc(fresh & ((1u << lane) - 1u))] = entry;
          queued += __popc(fresh);
          if (queued < 32 && !drained) continue;
          __syncwarp();
          // one child per lane: the queue's first 32
#pragma unroll 1
          while (queued >= 32 || (drained && queued > 0)) {
            const int n = queued < 32 ? queued : 32;
            entry = A.queue[lane];
            const unsigned later = A.queue[32 + lane];
            const unsigned from = entry >> 10, c = entry & 1023u;
            bool child = lane < n;
            uint2 it = item[child ? from : 0u];
            const int gid = (int)(it.y >> 30);
            const GuidedGroup &T = A.group[gid];
            GuidedBest best;
            best.key = kNone;
            best.cost = 0xffffffffu;
            Path path = none;
            if (child && d) {
              it.x ^= __ldg(T.hcol + c);
              uint32_t up = it.y;
#pragma unroll 1
              for (int e = d - 1; e > 0; --e) {
                push_col(path, (up >> 10) & 1023u);
                up = item[(up >> 20) & 1023u].y;
              }
              child = !in_path(path, c);
            }
            if (child && ((probes >> (G * gid)) & 1u))
              guided_probe<MLK>(T, T.am[i], path, d ? d - 1 : 0, d ? c : kNoCol, it.x, best);
            unsigned hit = __ballot_sync(kFull, best.key != kNone);
#pragma unroll 1
            for (; hit; hit &= hit - 1u) {  // rare: each match to its group's lanes
              const int src = __ffs((int)hit) - 1;
              const unsigned long long k2 = __shfl_sync(kFull, best.key, src);
              const uint32_t o2 = __shfl_sync(kFull, best.cost, src);
              if (__shfl_sync(kFull, gid, src) == g) {
                const bool less = !ml ? k2 < bkey
                                      : o2 < bcost || bkey == kNone ||
                                            (o2 == bcost && ml_set_before(llr, k2, bkey, w));
                if (less) {
                  bkey = k2;
                  bcost = o2;
                }
              }
            }
            const bool push = d && child && ((pushes >> (G * gid)) & 1u);
            if (__any_sync(kFull, push)) {
              bool keep = push;
              if (keep) {
                const Resid r = residual(T.sw, T.cols, T.wide != 0, path, d - 1, c);
                it.y = ((unsigned)gid << 30) | (from << 20) | (c << 10) | lowest_row(r);
                keep = ones_of(r) <= T.limit;
              }
              const unsigned kept = __ballot_sync(kFull, keep);
              const int at = top + __popc(kept & ((1u << lane) - 1u));
              top += __popc(kept);
              if (top > kGuidedItems) return 0;
              if (keep) item[at] = it;
            }
            A.queue[lane] = later;  // (all lanes have read theirs: the ballots above)
            queued -= n;
            __syncwarp();
          }
        }
        __syncwarp();
        if (d) {
          lo = hi;
          hi = top;
        }
        if (act && bkey != kNone && (!ml || !wn.w || bcost < wn.cost)) {
          wn.w = w;
          wn.key = bkey;
          wn.cost = bcost;
          if (!ml) go = false;
        }
        if (lo == hi && d && !wn.w) go = false;  // nothing left to extend
      }
      run = wn.w ? 0u : rest;
      rest = 0u;
    }

    // ---- the candidates the iteration reports ------------------------------------------
    const unsigned long long c15 = __shfl_sync(kFull, upto, gb + 5);
    const unsigned long long c6 = __shfl_sync(kFull, upto, gb + 6) - c15;
    const unsigned long long before = __shfl_sync(kFull, upto, gb + (wn.w ? wn.w - 1 : 0));
    unsigned long long total = __shfl_sync(kFull, upto, gb + wmax);
    unsigned long long upto_hit = __shfl_sync(kFull, upto, gb + (ml ? wn.w_done & 7 : wn.w));
    if (prob) {
      total = 0;
      bool past = false;  // the winner's phase is behind
#pragma unroll 1
      for (int k = 0; on && k < cd.num_phases; ++k) {
        const int pid = order[k];
        const unsigned long long n = pid == 0 ? c15 : (pid == 1 && tam >= 6 ? c6 : 0ull);
        total += n;
        const bool mine = wn.w && ((pid == 0 && wn.w <= 5) || (pid == 1 && wn.w == 6));
        // the phases before the winner's, and for the CPU branch the weights before it, for
        // the GPU branch the whole phase (grand_decoder.cu:1006)
        if (wn.w && !past) tested += mine && cpu ? (pid == 0 ? before : 0ull) : n;
        past = past || mine;
      }
    }
    if (on) {
      heavy |= total > (1ull << b.light_max_log2) || tam > kLightTam || tam * cd.nwp > kLightWords;
      hib = gpu ? (hib == -1 ? 1 : 0) : -1;
      if (!wn.w) tested += total;
      else if (ml) tested += cpu ? upto_hit : total;
      else if (!prob) tested += cpu ? before : total;  // grand_decoder.cu:1303-1304
    }
    const bool ranked = on && wn.w && !ml && cpu;
    if (__any_sync(kFull, ranked)) {
      // rank + 1 of the set among its weight's candidates (grand_decoder.cu:547-548)
      unsigned long long after = 0ull;
      if (ranked && gl < wn.w) {
        const unsigned c = set_col(wn.key, wn.w, gl);
        int idx = __popc(am[c >> 5] & ((1u << (c & 31u)) - 1u));
#pragma unroll 1
        for (int q = 0; q < (int)(c >> 5); ++q) idx += __popc(am[q]);
        const unsigned long long *u = b.upto + 8 * (tam - 1 - idx) + (wn.w - gl);
        after = __ldg(u) - __ldg(u - 1);
      }
#pragma unroll 1
      for (int o = 1; o < 8; o <<= 1) after += __shfl_xor_sync(kFull, after, o);
      after = __shfl_sync(kFull, after, gb);
      if (ranked) tested += upto_hit - before - after;
    }
    if (on && wn.w) found = i + 1;
  }
  tp = prof_lap(b, kProfShotLight, tp);

  // ---- the result --------------------------------------------------------------------
  const bool dem = cd.family == kDem;
  const int shot = F.shot[j];
  const bool errs = cd.input_kind == kInErrors;
  bool differs = false;
  if (live && found) {
    if (dem) {  // decoded logical flips vs the supplied true flips (grand_decoder.cu:1623-1644)
      if (gl < cd.nlw) {
        uint32_t le = 0u;
#pragma unroll 1
        for (int k = 0; k < wn.w; ++k)
          le ^= __ldg(cd.lcols + set_col(wn.key, wn.w, k) * (unsigned)cd.nlw + (unsigned)gl);
        differs = le != row[kRowLog + gl];
      }
    } else if (errs) {  // grand_decoder.cu:1362: as many columns, and each of them supplied
      const int at = F.at[j];
      differs = at < 0 || (int)row[kRowWeight] != wn.w;
      if (!differs && gl < wn.w) {
        const int c = at + (int)set_col(wn.key, wn.w, gl);
        differs = !((F.bits[c >> 5] >> (c & 31)) & 1u);
      }
    }
  }
  const bool told = ((__ballot_sync(kFull, differs) >> gb) & kGroup) != 0u;
  bool is_equal = live && found && !dem && errs && !told;
  bool degenerate = is_equal || (live && found && dem && !told);
  {
    // a supplied error that differs (or whose bits are not at hand): a group at a time, by
    // the whole warp
    unsigned todo = __ballot_sync(kFull, gl == 0 && told && !dem);
#pragma unroll 1
    for (; todo; todo &= todo - 1u) {
      const int src = __ffs((int)todo) - 1;
      const int e2 = __shfl_sync(kFull, entry, src);
      const int w2 = __shfl_sync(kFull, wn.w, src);
      const unsigned long long k2 = __shfl_sync(kFull, wn.key, src);
      const FastArea &F2 =
          *reinterpret_cast<const FastArea *>(reinterpret_cast<char *>(areas) + (e2 >> 8) * area_step);
      const int j2 = e2 & 255;
      const DevCode &cd2 = b.codes[F2.code[j2]];
      const uint32_t delta = set_word(k2, w2) ^ error_word(b, cd2, F2, F2.at[j2], F2.shot[j2]);
      const bool eq = __all_sync(kFull, delta == 0u);
      const bool deg2 = eq || in_row_space(cd2, delta);
      if (gb == src) {
        is_equal = eq;
        degenerate = deg2;
      }
    }
  }
  const int ow = live ? (int)row[kRowWeight] : 0;
  __syncwarp();  // every lane has read the open shot's words
  if (live && gl == 0) {
    const unsigned long long now = global_ns();
    const unsigned long long a = (unsigned long long)__double_as_longlong(1e-6 * (double)(t_counts - t_start));
    const unsigned long long s = (unsigned long long)__double_as_longlong(1e-6 * (double)(now - t_counts));
    const unsigned long long t =
        found ? (unsigned long long)__double_as_longlong(1e-6 * (double)(now - t_start)) : 0ull;
    row[0] = found ? 1u : 0u;
    row[1] = (uint32_t)wn.w;
    row[2] = (uint32_t)ow;
    row[3] = degenerate ? 1u : 0u;
    row[4] = is_equal ? 1u : 0u;
    row[5] = (uint32_t)tam;
    row[6] = (uint32_t)tested;
    row[7] = (uint32_t)(tested >> 32);
    row[8] = (uint32_t)hib;
    row[9] = (uint32_t)(found ? found : passes);
    row[10] = (uint32_t)a;
    row[11] = (uint32_t)(a >> 32);
    row[12] = (uint32_t)s;
    row[13] = (uint32_t)(s >> 32);
    row[14] = row[15] = 0u;
    row[16] = (uint32_t)t;
    row[17] = (uint32_t)(t >> 32);
    F.key[j] = wn.key;
    F.state[j] = 1;
    if (b.ml_cost) b.ml_cost[shot] = found && ml ? key_cost(wn.cost) : 0.0f;
  }
  __syncwarp();
  prof_lap(b, kProfShotFinish, tp);
  int ret = 0;
#pragma unroll 1
  for (int k = 0; k < 32 / G; ++k) {
    if (k < cnt) ret |= 1 << k;
    ret |= __shfl_sync(kFull, live && heavy ? 1 : 0, k * G) << (8 + k);
  }
  return ret;
}

}  // namespace grand
