// grand_guided.cuh -- the guided search of one shot by one warp (sm_103a).
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
// Levels.  The partial sets of one size lie side by side in shared memory ("items":
// the item extended and the column added, the residual's sketch and lowest row).  Level d extends the
// items of d - 1 columns by one: lanes take (item, neighbour) pairs, so a level
// of n items is n * deg / 32 steps whatever the shape of the tree; each new set
// probes the sketch filter for its last column (weight d + 1) and, while larger
// weights remain, is kept for the next level.  A level that outgrows the area
// gives the shot to the general path.
//
// The flagged-check counts (upstream grand_decoder.cu:67-81, 406-416) are formed
// from the rows: lane q holds mask word q of the columns, the rows of H selected by
// the syndrome are added into 3-bit counters kept as bit slices, and a column is
// active in iteration i when at most i of its rows are missing from the syndrome
// (its count, with the irregular offset, reaches max_soma - i).
//
// What bounds it: latency and the instruction caches.  A shot's work is some hundred
// instructions in a chain of L1 round trips (row words, adjacency, columns, filter),
// run once per shot by warps that are all somewhere else in it, so the code is
// kept small: loops stay rolled, column widths are a run-time choice and the rare
// parts are out of line.  Against the prefix-lookup search in Jobs (grand_lookup.cuh)
// that did this before: 20000 noisy [[288]] shots, W = 4, 957 -> 92 us; 8192 random
// detector records of the 120 x 720 DEM 562 -> 40 us.
#pragma once

#include "grand_kernels.cuh"

namespace grand {

// x: the residual's sketch; y: the item it extends (10 bits), the column added (10) and
// the residual's lowest row (10, kNoRow: zero).
struct alignas(16) GuidedArea {
  uint2 item[kGuidedItems];
  uint32_t sw[8];                // the syndrome, zero past nw
  uint32_t am[32];               // the searched iteration's active columns
  uint8_t rows[kGuidedMaxRows + 4];  // the syndrome's set rows, ascending, padded with R
};
constexpr unsigned kNoRow = 1023u;
static_assert(kGuidedItems <= 1024 && kGuidedMaxCols <= 1024 && kGuidedMaxRows < (int)kNoRow,
              "an item's fields have 10 bits each");

__device__ __forceinline__ uint32_t warp_xor(uint32_t v) {
#ifdef GRAND_HOST_EMULATION
  for (int o = 16; o > 0; o >>= 1) v ^= __shfl_xor_sync(kFull, v, o);
  return v;
#else
  return __reduce_xor_sync(kFull, v);
#endif
}
__device__ __forceinline__ int warp_add(int v) {
#ifdef GRAND_HOST_EMULATION
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
  return v;
#else
  return __reduce_add_sync(kFull, v);
#endif
}

// One code's tables and the search's state, uniform over the warp.
struct GuidedView {
  const uint32_t *cols, *filt, *tab;
  const uint16_t *adj;
  const uint32_t *hcol;
  const float *llr;          // nullptr: first-hit search
  uint32_t tab_mask;
  unsigned long long magic;  // ceil(2^32 / deg): p * magic >> 32 = p / deg for p < 2^26
  int deg, max_cw, m;
  bool wide;                 // more than 128 rows: columns of eight words
};

// A residual syndrome: the second half is used by codes of more than 128 rows (wide).
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

__device__ __forceinline__ unsigned set_col(unsigned long long key, int w, int e) {
  return (unsigned)(key >> (10 * (w - 1 - e))) & 1023u;
}

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
__device__ __forceinline__ void guided_probe(const GuidedArea &G, const GuidedView &v, const Path &p,
                                             int d, unsigned c, uint32_t h, GuidedBest &best) {
  const uint32_t f = h >> (32 - kGuidedF);
  if (!((__ldg(v.filt + (f >> 5)) >> (f & 31u)) & 1u)) return;
  uint32_t i = h & v.tab_mask;
#pragma unroll 1
  for (uint32_t guard = 0; guard <= v.tab_mask; ++guard) {
    const uint2 e = __ldg(reinterpret_cast<const uint2 *>(v.tab) + i);
    const unsigned j = e.y & 0xffffu;
    if (j == kNoCol) return;
    if (e.x == h && j != c && !in_path(p, j) && ((G.am[j >> 5] >> (j & 31u)) & 1u))
      best = guided_match<MLK>(G.sw, v.cols, v.wide, v.llr, p, d, c, j, best);
    i = (i + 1u) & v.tab_mask;
  }
}

// What the search found (uniform over the warp).
struct GuidedWinner {
  int w;                    // 0: nothing
  unsigned long long key;   // its columns, in list order
  uint32_t cost;            // ML cost key
  int w_done;               // ML: last weight searched (the bound may stop it early)
};

// FP32 sum of the w smallest LLRs of the active columns (the bound of weight w):
// upstream's prefix sums add them in ascending order.
static __device__ __noinline__ float ml_prefix(const uint32_t *am, const float *llr, int m, int w) {
  const int lane = threadIdx.x & 31;
  float sum = 0.0f;
  unsigned long long last = 0ull;  // {LLR key, column} of the smallest taken so far, plus one
#pragma unroll 1
  for (int e = 0; e < w; ++e) {
    unsigned long long best = kNone;
#pragma unroll 1
    for (int c0 = 0; c0 < m; c0 += 32) {
      const int c = c0 + lane;
      if ((am[c0 >> 5] >> lane) & 1u) {  // bits past m are 0
        const uint32_t u = __float_as_uint(__ldg(llr + c));
        const uint32_t k = (u & 0x80000000u) ? ~u : (u | 0x80000000u);
        const unsigned long long x = ((unsigned long long)k << 32) | (unsigned)c;
        if (x >= last && x < best) best = x;
      }
    }
    best = warp_min_u64(best);
    if (best == kNone) break;
    const uint32_t k = (uint32_t)(best >> 32);
    sum = __fadd_rn(sum, __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k));
    last = best + 1ull;
  }
  return sum;
}

// Weights w_first .. w_last of the active set G.am in ascending order, to the first
// weight with a match (ML: to the bound).  hs: the syndrome's sketch, ones / row0: its
// number of set rows and its lowest.  Returns false when a level does not fit.
//
// Weight w is searched while its level is formed: every item of w - 2 columns is
// extended by one (items lo .. hi), each new set probes for its last column, and,
// while larger weights remain, sets that can still reach weight w_last are kept from
// index hi on.
template <bool MLK>
__device__ __forceinline__ bool guided_search(GuidedArea &G, const GuidedView &v, uint32_t hs,
                                              int ones, unsigned row0, int w_first, int w_last,
                                              GuidedWinner &wn) {
  const int lane = threadIdx.x & 31;
  const bool ml = MLK && v.llr != nullptr;
  wn.w = 0;
  wn.key = kNone;
  wn.cost = 0xffffffffu;
  wn.w_done = w_last;
  if (ones > v.max_cw * w_last) return true;  // no w_last columns hold that many rows
  const Path none{0xffffffffu, 0xffffffffu};
  if (lane == 0) G.item[0] = make_uint2(hs, row0);
  __syncwarp();
  int lo = 0, hi = 1;
#pragma unroll 1
  for (int w = 1; w <= w_last; ++w) {
    if (MLK && ml && wn.w && ml_prefix(G.am, v.llr, v.m, w) >= key_cost(wn.cost)) {
      wn.w_done = w - 1;
      return true;
    }
    GuidedBest best;
    best.key = kNone;
    best.cost = 0xffffffffu;
    const int d = w - 1;  // columns of the sets formed
    const bool probe = w >= w_first, push = w < w_last;
    if (d == 0) {
      if (probe && lane == 0) guided_probe<MLK>(G, v, none, 0, kNoCol, hs, best);
    } else {
      const int pairs = (hi - lo) * v.deg;
      int top = hi;
      int z = -1;  // an item of residual zero being extended (by every active column), -1: none yet
      unsigned zeros = 0u;
      // steps of 32 (item, neighbour) pairs, then, for each item without a row to
      // follow, steps of 32 columns
#pragma unroll 1
      for (int p0 = 0;; p0 += 32) {
        int i = lo;
        unsigned c = kNoCol;
        uint2 it = make_uint2(0u, 0u);
        if (z < 0 && p0 < pairs) {
          const int p = p0 + lane;
          if (p < pairs) {
            const int q = (int)(((unsigned long long)(unsigned)p * v.magic) >> 32);
            i = lo + q;
            it = G.item[i];
            const unsigned row = it.y & 1023u;
            if (row != kNoRow) c = __ldg(v.adj + row * (unsigned)v.deg + (unsigned)(p - q * v.deg));
            else zeros = 1u;
          }
        } else {
          if (z < 0 || p0 >= v.m) {
            if (z < 0 && !__any_sync(kFull, zeros != 0u)) break;  // (ML, or weights out of order)
            z = z < 0 ? lo : z + 1;
            while (z < hi && (G.item[z].y & 1023u) != kNoRow) ++z;
            if (z >= hi) break;
            p0 = 0;
          }
          i = z;
          it = G.item[z];
          if (p0 + lane < v.m) c = (unsigned)(p0 + lane);
        }
        // one child per lane: column c after item i, if active and not in it
        bool live = c != kNoCol && ((G.am[(c >> 5) & 31u] >> (c & 31u)) & 1u);
        Path path = none;
        if (live) {
          it.x ^= __ldg(v.hcol + c);
          uint32_t up = it.y;
#pragma unroll 1
          for (int e = d - 1; e > 0; --e) {
            push_col(path, (up >> 10) & 1023u);
            up = G.item[up >> 20].y;
          }
          live = !in_path(path, c);
          if (live && probe) guided_probe<MLK>(G, v, path, d - 1, c, it.x, best);
        }
        if (push) {
          if (live) {
            const Resid r = residual(G.sw, v.cols, v.wide, path, d - 1, c);
            it.y = ((unsigned)i << 20) | (c << 10) | lowest_row(r);
            live = ones_of(r) <= v.max_cw * (w_last - d);
          }
          const unsigned keep = __ballot_sync(kFull, live);
          const int at = top + __popc(keep & ((1u << lane) - 1u));
          top += __popc(keep);
          if (top > kGuidedItems) return false;
          if (live) G.item[at] = it;
        }
      }
      __syncwarp();
      lo = hi;
      hi = top;
    }
    if (__any_sync(kFull, best.key != kNone)) {
      if (!ml) {
        wn.w = w;
        wn.key = warp_min_u64(best.key);
        return true;
      }
      const uint32_t o = __reduce_min_sync(kFull, best.cost);
      unsigned who = __ballot_sync(kFull, best.key != kNone && best.cost == o);
      unsigned long long key = __shfl_sync(kFull, best.key, __ffs((int)who) - 1);
#pragma unroll 1
      for (who &= who - 1u; who; who &= who - 1u) {
        const unsigned long long k2 = __shfl_sync(kFull, best.key, __ffs((int)who) - 1);
        if (ml_set_before(v.llr, k2, key, w)) key = k2;
      }
      if (!wn.w || o < wn.cost) {
        wn.w = w;
        wn.key = key;
        wn.cost = o;
      }
    }
    if (lo == hi && w > 1 && !wn.w) break;  // nothing left to extend
  }
  return true;
}

// x added to the counters of each bit position.
__device__ __forceinline__ void add_bits(uint32_t x, uint32_t &c0, uint32_t &c1, uint32_t &c2) {
  const uint32_t t = c0 & x;
  c0 ^= x;
  c2 ^= c1 & t;
  c1 ^= t;
}

// Exclusive prefix sum over the lanes.
__device__ __forceinline__ int lanes_before(int v) {
  const int lane = threadIdx.x & 31;
  int sum = v;
#pragma unroll 1
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(kFull, sum, o);
    if (lane >= o) sum += u;
  }
  return sum - v;
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

// out[0 .. n) = the bits of word `lane` of a vector, one byte each.
__device__ __forceinline__ void bits_to_bytes(unsigned char *out, int n, uint32_t word) {
  const int lane = threadIdx.x & 31;
#pragma unroll 1
  for (int c0 = 0; c0 < n; c0 += 32) {
    const uint32_t w = __shfl_sync(kFull, word, c0 >> 5);
    if (c0 + lane < n) out[c0 + lane] = (unsigned char)((w >> lane) & 1u);
  }
}

// One shot, start to finish, by one warp: the threshold iterations in upstream's order
// (grand_decoder.cu:1284-1343) until one has a match, and the shot's result.
// s_lane: syndrome word `lane` (0 past nw), not all zero; hs: its sketch; eb_lane: word
// `lane` of the supplied error (CSS) or of the true logical flips (DEM), 0 past the
// last.  Returns 1 when done, 2 when done and past the light budget, 0 when the shot
// needs the general path (nothing has been written).
template <bool MLK>
__device__ __forceinline__ int guided_shot(const DevBatch &b, const DevCode &cd, int shot, GuidedArea &G,
                                        uint32_t s_lane, uint32_t hs, uint32_t eb_lane,
                                        int original_weight, unsigned long long t_start) {
  const int lane = threadIdx.x & 31;
  const bool ml = MLK && cd.variant == kMl;
  const int mw = cd.mw;
  unsigned long long tp = b.profile ? global_ns() : 0ull;

  // ---- the syndrome and its rows ------------------------------------------------
  if (lane < 8) G.sw[lane] = s_lane;
  int ones = 0;
#pragma unroll 1
  for (int k = 0; k < cd.nw; ++k) {
    const uint32_t word = __shfl_sync(kFull, s_lane, k);
    if ((word >> lane) & 1u) G.rows[ones + __popc(word & ((1u << lane) - 1u))] = (uint8_t)(32 * k + lane);
    ones += __popc(word);
  }
  if (lane < 4) G.rows[ones + lane] = (uint8_t)cd.R;  // the row of zeros behind the table's
  __syncwarp();

  // ---- counts, bit-sliced: lane q the columns of mask word q ----------------------
  const int L = cd.max_soma < kMaxIters ? cd.max_soma : kMaxIters;
  uint32_t am0 = 0u, am1 = 0u, am2 = 0u;
  {
    // up to 8 mask words: four groups of lanes share the rows and add their counts up;
    // up to 16: two groups; the list ends with rows of zeros
    const int split = mw <= 8 ? 4 : (mw <= 16 ? 2 : 1);
    const int q = lane & (32 / split - 1);
    const int step = 4 * split, part = lane / (32 / split);
    const uint32_t *rows = cd.g_rows + (q < mw ? q : 0);
    uint32_t c0 = 0u, c1 = 0u, c2 = 0u;
#pragma unroll 1
    for (int i = 4 * part; i < ones; i += step) {
      const uchar4 r = *reinterpret_cast<const uchar4 *>(G.rows + i);
      const uint32_t x0 = __ldg(rows + (int)r.x * mw), x1 = __ldg(rows + (int)r.y * mw),
                     x2 = __ldg(rows + (int)r.z * mw), x3 = __ldg(rows + (int)r.w * mw);
      add_bits(x0, c0, c1, c2);
      add_bits(x1, c0, c1, c2);
      add_bits(x2, c0, c1, c2);
      add_bits(x3, c0, c1, c2);
    }
    __syncwarp();
#pragma unroll 1
    for (int o = 32 / split; o < 32; o <<= 1) {
      const uint32_t y0 = __shfl_xor_sync(kFull, c0, o), y1 = __shfl_xor_sync(kFull, c1, o),
                     y2 = __shfl_xor_sync(kFull, c2, o);
      const uint32_t t0 = c0 & y0, t1 = (c1 & y1) | (t0 & (c1 ^ y1));
      c2 ^= y2 ^ t1;
      c1 ^= y1 ^ t0;
      c0 ^= y0;
    }
    if (lane < mw) {
      const uint32_t w0 = __ldg(cd.g_cw + lane), w1 = __ldg(cd.g_cw + mw + lane),
                     w2 = __ldg(cd.g_cw + 2 * mw + lane);
      // missing = weight - count, bit by bit; zero columns are never active
      const uint32_t nz = w0 | w1 | w2;
      const uint32_t m0 = w0 ^ c0, b0 = ~w0 & c0;
      const uint32_t m1 = w1 ^ c1 ^ b0, b1 = (~w1 & c1) | (~(w1 ^ c1) & b0);
      const uint32_t m2 = w2 ^ c2 ^ b1;
      am0 = nz & ~(m0 | m1 | m2);
      am1 = nz & ~(m1 | m2);
      am2 = nz & ~(m2 | (m1 & m0));
    }
  }
  const unsigned long long t_counts = global_ns();
  tp = prof_lap(b, kProfShotCounts, tp);

  GuidedView v;
  v.cols = cd.g_cols;
  v.filt = cd.g_filt;
  v.tab = cd.g_tab;
  v.adj = cd.g_adj;
  v.hcol = cd.g_hcol;
  v.llr = ml ? cd.llr : nullptr;
  v.tab_mask = cd.g_tab_mask;
  v.deg = cd.g_deg;
  v.magic = cd.g_magic;
  v.max_cw = cd.g_max_cw;
  v.m = cd.m;
  v.wide = cd.g_gs == 8;

  // ---- the iterations --------------------------------------------------------------
  const bool prob = cd.variant == kProb;
  GuidedWinner wn;
  wn.w = 0;
  int tam = 0, tam_old = 0, passes = 0, hib = -2, heavy = 0, found = 0;
  unsigned long long tested = 0;
#pragma unroll 1
  for (int i = 0; i < L && !found; ++i) {
    passes = i + 1;
    uint32_t am = am0;
    am0 = am1;
    am1 = am2;
    const int n_act = warp_add(__popc(am));
    tam = n_act;
    if (cd.family == kDem) {  // grand_decoder.cu:1550-1554
      if (tam > cd.cap) tam = tam_old;
      else tam_old = tam;
    }
    if (tam <= 0) continue;
    const bool gpu = (tam > cd.thr && tam <= cd.cap && cd.mode == 1) || cd.mode == 0;
    const bool cpu = !gpu && ((tam <= cd.thr && cd.mode == 1) || cd.mode == -1);
    if (!gpu && !cpu) continue;
    if (tam < n_act) {  // the first tam columns of the larger set (the cap rule)
      int left = tam - lanes_before(__popc(am));
      uint32_t rest = am;
      am = 0u;
#pragma unroll 1
      for (; rest && left > 0; --left) {
        am |= rest & (0u - rest);
        rest &= rest - 1u;
      }
    }
    G.am[lane] = am;
    __syncwarp();

    // candidate counts: lane w holds those of weights 1 .. w
    unsigned long long upto = lane >= 1 ? ncr(b.ncr, tam, lane) : 0ull;
#pragma unroll 1
    for (int o = 1; o < 8; o <<= 1) {
      const unsigned long long u = __shfl_up_sync(kFull, upto, o);
      if (lane >= o) upto += u;
    }
    const unsigned long long c15 = __shfl_sync(kFull, upto, 5);
    const unsigned long long c6 = __shfl_sync(kFull, upto, 6) - c15;
    // the weights searched (bit w), in one ascending run or weight 6 (run) before the others
    unsigned long long total = 0;
    unsigned ws = 0u, run;
    int mi = 0;
    if (prob) {
      mi = cd.n_masks - 1;  // grand_decoder.cu:754-762
#pragma unroll 1
      for (int q = 0; q < cd.n_masks; ++q)
        if (tam <= cd.mask_tam_upper[q]) {
          mi = q;
          break;
        }
      run = 0u;
#pragma unroll 1
      for (int k = 0; k < cd.num_phases; ++k) {
        const int pid = cd.mask_order[mi][k];
        if (pid == 0) {
          total += c15;
          ws |= (2u << (tam < 5 ? tam : 5)) - 2u;
        } else if (pid == 1 && tam >= 6) {
          total += c6;
          if (!ws) run = 64u;
          ws |= 64u;
        }
      }
      if (!run) run = ws;
    } else {
      const int wmax = cd.Wc < tam ? cd.Wc : tam;
      total = __shfl_sync(kFull, upto, wmax);
      run = ws = (2u << wmax) - 2u;
    }
    heavy |= total > (1ull << b.light_max_log2) || tam > kLightTam || tam * cd.nwp > kLightWords;

#pragma unroll 1
    for (unsigned rest = ws & ~run; run; run = rest, rest = 0u) {
      if (!guided_search<MLK>(G, v, hs, ones, G.rows[0], __ffs((int)run) - 1, 31 - __clz((int)run), wn))
        return 0;
      if (wn.w) break;
    }
    hib = gpu ? (hib == -1 ? 1 : 0) : -1;
    if (!wn.w) {
      tested += total;
      continue;
    }
    found = i + 1;
    // the candidates the winning iteration reports
    if (ml) {
      tested += cpu ? __shfl_sync(kFull, upto, wn.w_done) : total;
    } else if (prob) {
      // the phases before the winner's, and for the CPU branch the weights before it,
      // for the GPU branch the whole phase (grand_decoder.cu:1006)
#pragma unroll 1
      for (int k = 0; k < cd.num_phases; ++k) {
        const int pid = cd.mask_order[mi][k];
        const bool hit = (pid == 0 && wn.w <= 5) || (pid == 1 && wn.w == 6);
        if (hit && cpu) {
          if (pid == 0) tested += __shfl_sync(kFull, upto, wn.w - 1);
          break;
        }
        if (pid == 0) tested += c15;
        if (pid == 1) tested += c6;
        if (hit) break;
      }
    } else {
      tested += cpu ? __shfl_sync(kFull, upto, wn.w - 1) : total;  // grand_decoder.cu:1303-1304
    }
    if (!ml && cpu) {
      // rank + 1 of the set among its weight's candidates (grand_decoder.cu:547-548)
      const int pre = lanes_before(__popc(am));
      const unsigned c = lane < wn.w ? set_col(wn.key, wn.w, lane) : 0u;
      const int idx = __shfl_sync(kFull, pre, (int)(c >> 5)) + __popc(G.am[c >> 5] & ((1u << (c & 31u)) - 1u));
      unsigned long long after = lane < wn.w ? ncr(b.ncr, tam - 1 - idx, wn.w - lane) : 0ull;
#pragma unroll 1
      for (int o = 4; o > 0; o >>= 1) after += __shfl_xor_sync(kFull, after, o);
      tested += __shfl_sync(kFull, upto, wn.w) - __shfl_sync(kFull, upto, wn.w - 1) -
                __shfl_sync(kFull, after, 0);
    }
  }
  tp = prof_lap(b, kProfShotLight, tp);

  // ---- the result --------------------------------------------------------------------
  uint32_t e = 0u;   // word `lane` of the decoded error
  uint32_t le = 0u;  // and of its logical flips (DEM)
  const bool dem = cd.family == kDem;
#pragma unroll 1
  for (int k = 0; k < wn.w; ++k) {
    const unsigned c = set_col(wn.key, wn.w, k);
    if ((int)(c >> 5) == lane) e |= 1u << (c & 31u);
    if (dem && lane < cd.nlw) le ^= __ldg(cd.lcols + c * (unsigned)cd.nlw + (unsigned)lane);
  }
  int degenerate = 0, is_equal = 0;
  if (found && dem) {
    // decoded logical flips vs the supplied true flips (grand_decoder.cu:1623-1644)
    degenerate = __all_sync(kFull, le == eb_lane) ? 1 : 0;
  } else if (found && cd.input_kind == kInErrors) {
    is_equal = __all_sync(kFull, e == eb_lane) ? 1 : 0;  // grand_decoder.cu:1362
    degenerate = is_equal || in_row_space(cd, e ^ eb_lane) ? 1 : 0;
  }
  if (dem && b.dec_log) bits_to_bytes(b.dec_log + (size_t)shot * cd.n_logicos, cd.n_logicos, le);
  if (b.dec_err) bits_to_bytes(b.dec_err + (size_t)shot * cd.m, cd.m, e);
  // the 72-byte result as 18 words, one per lane (finish_shot's layout and times)
  const unsigned long long now = global_ns();
  const unsigned long long dt = lane < 12 ? t_counts - t_start : lane < 14 ? now - t_counts
                                : lane < 16 || !found ? 0ull : now - t_start;
  const unsigned long long bits = (unsigned long long)__double_as_longlong(1e-6 * (double)dt);
  uint32_t x = (lane & 1) ? (uint32_t)(bits >> 32) : (uint32_t)bits;
  x = lane == 9 ? (uint32_t)(found ? found : passes) : x;
  x = lane == 8 ? (uint32_t)hib : x;
  x = lane == 7 ? (uint32_t)(tested >> 32) : x;
  x = lane == 6 ? (uint32_t)tested : x;
  x = lane == 5 ? (uint32_t)tam : x;
  x = lane == 4 ? (uint32_t)is_equal : x;
  x = lane == 3 ? (uint32_t)degenerate : x;
  x = lane == 2 ? (uint32_t)original_weight : x;
  x = lane == 1 ? (uint32_t)wn.w : x;
  x = lane == 0 ? (found ? 1u : 0u) : x;
  if (lane < 18) reinterpret_cast<uint32_t *>(b.results + shot)[lane] = x;
  if (lane == 0) {
    if (b.ml_cost) b.ml_cost[shot] = found && ml ? key_cost(wn.cost) : 0.0f;
    if (b.deferred) b.deferred[shot] = 0;
  }
  __syncwarp();
  prof_lap(b, kProfShotFinish, tp);
  return heavy ? 2 : 1;
}

}  // namespace grand
