// grand_prep.cuh -- a code's tables built on the device from its check matrix, by one block
// (sm_103a): the packed columns, weights and sketches, and the guided search's tables
// (grand_guided_tables.h), for the entry point that may keep nothing between calls.
//
// The matrix is read once, coalesced, into bit rows in shared memory; everything else is
// formed from those: columns by walking the rows' bits, a column per thread; the row
// lists by ballot; the sketch table in the same memory afterwards; solo columns
// (grand_solo.h) by counting, bit-sliced, how many of a column's rows hold each other
// column.  Bound by the latency of that sequence of block-wide steps:
// 16.5 us for the [[108,8,10]] code (20.2 with divisions in the loops, the solo test on
// columns in global memory and the descriptor copied by one thread).
#pragma once

#include "grand_kernels.cuh"

namespace grand {

constexpr int kPrepMaxRows = 256, kPrepMaxCols = 1024;

// Offsets of the guided tables in their block, for the largest degree (words).
struct PrepLayout {
  int rows, cw, adj, cols, filt, tab, hcol, nib, total;
};
GRAND_HD inline PrepLayout prep_layout(int n, int m, int deg, int slots) {
  PrepLayout L;
  const int mw = (m + 31) / 32, gs = n <= 128 ? 4 : 8;
  L.rows = 0;
  L.cw = L.rows + (((n + 1) * mw + 3) & ~3);
  L.adj = L.cw + ((3 * mw + 3) & ~3);
  L.cols = L.adj + (((n * deg + 1) / 2 + 3) & ~3);
  L.filt = L.cols + m * gs;
  L.tab = L.filt + (1 << (kGuidedF - 5));
  L.hcol = L.tab + 2 * slots;
  L.nib = L.hcol + ((m + 3) & ~3);
  L.total = L.nib + nib_words(n);
  return L;
}
// Words the guided tables can take at the entry point's limits.
constexpr size_t kPrepWords = (kPrepMaxRows + 1) * 32 + 96 + kPrepMaxRows * kGuidedMaxDegree / 2 +
                              kPrepMaxCols * 8 + (1 << (kGuidedF - 5)) + 4 * kPrepMaxCols + kPrepMaxCols + 1024 + 64;

struct PrepShared {
  uint32_t bits[(kPrepMaxRows + 1) * 32];  // the rows, then the sketch table
  uint32_t filt[1 << (kGuidedF - 5)];
  uint32_t cw[3][32];
  unsigned long long crow[kPrepMaxCols];  // a column's rows, a byte each from the lowest up
  int deg, max_w, min_w, max_cw, even, nonbinary;
};

// tmpl: the descriptor but for what depends on H; solo_branch as for a code with solo
// columns.  guided: kPrepWords words.  clear: clear_words 64-bit control words, zeroed.
__global__ void __launch_bounds__(1024, 1) prep_kernel(const DevCode tmpl, const int *H, uint32_t *cols, int *colw,
                                                    uint32_t *hcol, uint32_t *guided, DevCode *out,
                                                    unsigned long long *clear, int clear_words) {
  __shared__ PrepShared S;
  const int n = tmpl.R, m = tmpl.m, mw = tmpl.mw, nw = tmpl.nw, nwp = tmpl.nwp;
  const int T = (int)blockDim.x, t = (int)threadIdx.x, lane = t & 31, warp = t >> 5, warps = T >> 5;
  const unsigned lt = (1u << lane) - 1u;
  for (int i = t; i < clear_words; i += T) clear[i] = 0ull;
  for (int i = t; i < (int)(sizeof(DevCode) / 8); i += T)
    reinterpret_cast<unsigned long long *>(out)[i] = reinterpret_cast<const unsigned long long *>(&tmpl)[i];
  for (int i = t; i < (1 << (kGuidedF - 5)); i += T) S.filt[i] = 0u;
  if (t < 32) {
    S.bits[n * mw + t < (kPrepMaxRows + 1) * 32 ? n * mw + t : 0] = 0u;  // the row of zeros
    S.cw[0][t] = S.cw[1][t] = S.cw[2][t] = 0u;
  }
  if (t == 0) {
    S.deg = S.max_cw = S.even = S.nonbinary = 0;
    S.max_w = -0x7fffffff - 1;
    S.min_w = 0x7fffffff;
  }
  __syncthreads();

  // ---- rows: words of all of them in one list, eight loads in flight per lane ----------
  int degree_seen = 0;
  bool odd_value = false;
  const int words = n * mw;
#pragma unroll 1
  for (int w0 = warp * 8; w0 < words; w0 += warps * 8) {
    int v[8];
    int r = w0 / mw, q = w0 - r * mw;
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int c = q * 32 + lane;
      v[u] = w0 + u < words && c < m ? __ldg(H + (size_t)r * m + c) : 0;
      if (++q == mw) {
        q = 0;
        ++r;
      }
    }
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const uint32_t b = __ballot_sync(kFull, v[u] != 0);
      if (lane == 0 && w0 + u < words) S.bits[w0 + u] = b;
      odd_value = odd_value || (v[u] != 0 && v[u] != 1);
    }
  }
  if (odd_value) S.nonbinary = 1;
  __syncthreads();
#pragma unroll 1
  for (int r = t; r < n; r += T) {
    int d = 0;
#pragma unroll 1
    for (int q = 0; q < mw; ++q) d += __popc(S.bits[r * mw + q]);
    degree_seen = d > degree_seen ? d : degree_seen;
  }
  if (degree_seen) atomicMax(&S.deg, degree_seen);
  __syncthreads();
  const int deg = S.deg;
  int slots = 2;
  while (slots < 2 * m) slots <<= 1;
  const bool small = !S.nonbinary && n <= kGuidedMaxRows && m <= kGuidedMaxCols && deg >= 1 && deg <= kGuidedMaxDegree;
  const PrepLayout L = prep_layout(n, m, small ? deg : 1, slots);
  const int gs = n <= 128 ? 4 : 8;

  // ---- columns ---------------------------------------------------------------------------
#pragma unroll 1
  for (int c0 = 0; c0 < m; c0 += T) {  // (uniform: whole warps ballot)
    const int c = c0 + t;
    uint32_t h = 0u;
    int ones = 0;
    unsigned long long rows = 0ull;
#pragma unroll 1
    for (int k = 0; k < (small ? gs : nwp); ++k) {
      uint32_t acc = 0u;
#pragma unroll 4
      for (int r = 32 * k; r < 32 * k + 32 && r < n; ++r)
        if (c < m) acc |= ((S.bits[r * mw + (c >> 5)] >> (c & 31)) & 1u) << (r & 31);
      if (c >= m) continue;
      if (k < nwp) cols[(size_t)c * nwp + k] = acc;
      if (small) guided[L.cols + c * gs + k] = acc;
#pragma unroll 1
      for (; acc; acc &= acc - 1u) {
        const int r = 32 * k + __ffs((int)acc) - 1;
        h ^= row_hash(r);
        if (ones < 8) rows |= (unsigned long long)r << (8 * ones);
        ++ones;
      }
    }
    int w = ones;
    if (c < m && S.nonbinary) {  // weights are sums of the entries
      w = 0;
#pragma unroll 1
      for (int r = 0; r < n; ++r) w += __ldg(H + (size_t)r * m + c);
    }
    if (c < m) {
      colw[c] = w;
      hcol[c] = h;
      if (small) guided[L.hcol + c] = h;
      S.crow[c] = rows;
      if (ones && !(ones & 1)) S.even = 1;
      atomicOr(&S.filt[(h >> (32 - kGuidedF)) >> 5], 1u << ((h >> (32 - kGuidedF)) & 31u));
    }
    {  // the block's extremes, one shared atomic per warp (weights biased to stay in order)
      const unsigned bias = 0x80000000u;
      const unsigned wu = (unsigned)w ^ bias;
      const unsigned hi = __reduce_max_sync(kFull, c < m ? wu : 0u);
      const unsigned lo = __reduce_min_sync(kFull, c < m ? wu : kFull);
      const unsigned oh = __reduce_max_sync(kFull, c < m ? (unsigned)ones : 0u);
      if (lane == 0 && c < m) {
        atomicMax(&S.max_w, (int)(hi ^ bias));
        atomicMin(&S.min_w, (int)(lo ^ bias));
        atomicMax(&S.max_cw, (int)oh);
      }
    }
#pragma unroll
    for (int b = 0; b < 3; ++b) {
      const uint32_t slice = __ballot_sync(kFull, c < m && ((ones >> b) & 1));
      if (lane == 0 && (c >> 5) < 32) S.cw[b][c >> 5] = slice;
    }
  }
  __syncthreads();
  const bool ok = small && S.max_cw >= 1 && S.max_cw <= kGuidedMaxColWeight;

  if (ok) {
    // ---- row lists, and what is copied as it is ------------------------------------------
    uint16_t *adj = reinterpret_cast<uint16_t *>(guided + L.adj);
#pragma unroll 1
    for (int r = warp; r < n; r += warps) {
      int base = 0;
#pragma unroll 1
      for (int q = 0; q < mw; ++q) {
        const uint32_t word = S.bits[r * mw + q];
        if ((word >> lane) & 1u) adj[r * deg + base + __popc(word & lt)] = (uint16_t)(32 * q + lane);
        base += __popc(word);
      }
      for (int k = base + lane; k < deg; k += 32) adj[r * deg + k] = (uint16_t)kNoCol;
    }
    for (int i = t; i < (n + 1) * mw; i += T) guided[L.rows + i] = S.bits[i];
    for (int i = t; i < nib_words(n); i += T) guided[L.nib + i] = nib_sketch(i);
    for (int i = t; i < 96; i += T)
      if ((i & 31) < mw) guided[L.cw + (i >> 5) * mw + (i & 31)] = S.cw[i >> 5][i & 31];
    for (int i = t; i < (1 << (kGuidedF - 5)); i += T) guided[L.filt + i] = S.filt[i];
  }
  // ---- solo columns: those whose rows hold no other column whole --------------------------
  // (a thread's answers as bits: at most kPrepMaxCols / 32 columns each)
  uint32_t solo = 0u;
  if (ok) {
#pragma unroll 1
    for (int c = t, k = 0; c < m; c += T, ++k) {
      uint32_t others = 0u;
      const unsigned long long rows = S.crow[c];
      const int own = c >> 5, bit = c & 31;
      const int weight = (int)(((S.cw[0][own] >> bit) & 1u) | (((S.cw[1][own] >> bit) & 1u) << 1) |
                               (((S.cw[2][own] >> bit) & 1u) << 2));
#pragma unroll 1
      for (int q = 0; q < mw; ++q) {
        uint32_t c0 = 0u, c1 = 0u, c2 = 0u;
#pragma unroll 1
        for (int e = 0; e < weight; ++e) {
          const uint32_t x = S.bits[(int)((rows >> (8 * e)) & 255u) * mw + q];
          const uint32_t y = c0 & x;
          c0 ^= x;
          c2 ^= c1 & y;
          c1 ^= y;
        }
        const uint32_t w0 = S.cw[0][q], w1 = S.cw[1][q], w2 = S.cw[2][q];
        uint32_t in = (w0 | w1 | w2) & ~((w0 ^ c0) | (w1 ^ c1) | (w2 ^ c2));
        if (q == own) in &= ~(1u << bit);
        others |= in;
      }
      if (weight && !others) solo |= 1u << k;
    }
  }
  __syncthreads();  // the rows' last use
  if (ok) {
    // ---- the sketch table ----------------------------------------------------------------
    uint32_t *tab = S.bits;
    for (int i = t; i < slots; i += T) tab[2 * i + 1] = kNoCol;
    __syncthreads();
#pragma unroll 1
    for (int c = t, k = 0; c < m; c += T, ++k) {
      const uint32_t h = guided[L.hcol + c];
      int i = (int)(h & (uint32_t)(slots - 1));
      const uint32_t mine = (uint32_t)c | ((solo >> k) & 1u ? kSoloFlag : 0u);
#pragma unroll 1
      for (int guard = 0; guard < slots && atomicCAS(&tab[2 * i + 1], (unsigned)kNoCol, mine) != kNoCol; ++guard)
        i = (i + 1) & (slots - 1);
      tab[2 * i] = h;
    }
    __syncthreads();
    for (int i = t; i < 2 * slots; i += T) guided[L.tab + i] = (i & 1) || tab[i + 1] != kNoCol ? tab[i] : 0u;
  }
  if (t == 0) {
    DevCode &d = *out;  // (the template's words were copied at the start)
    d.max_soma = S.max_w > 0 ? S.max_w : 0;
    d.regular = S.min_w == S.max_w ? 1 : 0;
    if (ok) {
      d.g_gs = gs;
      d.g_deg = deg;
      d.g_max_cw = S.max_cw;
      d.g_odd = S.even ? 0 : 1;
      d.g_tab_mask = (uint32_t)(slots - 1);
      d.g_words = L.total;
      d.g_magic = 0xffffffffull / (unsigned)deg + 1ull;
      d.g_rows = guided + L.rows;
      d.g_cw = guided + L.cw;
      d.g_cols = guided + L.cols;
      d.g_filt = guided + L.filt;
      d.g_tab = guided + L.tab;
      d.g_hcol = guided + L.hcol;
      d.g_nib = guided + L.nib;
      d.g_adj = reinterpret_cast<const uint16_t *>(guided + L.adj);
    } else {
      d.solo_branch = kSoloNone;
    }
  }
}

}  // namespace grand
