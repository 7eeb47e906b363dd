// grand_guided_tables.h -- a code's tables for the guided search (host side, built
// with the code tables; the search itself is grand_guided.cuh).
//
//   rows   R rows of H packed into mw = ceil(m/32) words (bit c of row r), then one of
//          zeros
//   cw     the column weights bit-sliced: bit c of cw[b * mw + (c >> 5)] is bit b of
//          column c's weight, b < 3
//   adj    the columns of each row, ascending, deg u16 per row (kNoCol past the
//          row's own degree)
//   cols   m columns packed into gs = 4 or 8 words
//   filt   a 2^kGuidedF-bit filter of the column sketches (one bit per column)
//   tab    the columns by sketch: open addressing, linear probing, {sketch, column}
//          pairs (column kNoCol = empty slot; kSoloFlag set for a solo column,
//          grand_solo.h), at most half full
//   hcol   the column sketches
//   nib    the sketches of four rows at a time: nib[16 i + v] is that of the rows 4i + b
//          with bit b of v set
//
// A code has them when its matrix is 0/1, with at most 255 rows, 1024 columns, 7
// ones per column and 64 per row: the search keeps a residual syndrome in 4 or 8
// registers and one mask word per lane, counts in 3 bits, and gains from rows
// that meet few columns.
#pragma once

#include <stdint.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "grand_common.h"
#include "grand_solo.h"

namespace grand {

struct GuidedTables {
  int gs = 0, deg = 0, max_cw = 0, odd = 1;
  uint32_t tab_mask = 0;
  // one block of words; the parts start at these word offsets (16-byte aligned)
  size_t total = 0, o_rows = 0, o_cw = 0, o_adj = 0, o_cols = 0, o_filt = 0, o_tab = 0, o_hcol = 0, o_nib = 0;
  std::vector<uint32_t> words;  // empty: the code has no guided search
};

// cols: m columns of nwp words; hcol: their sketches; binary: every entry of H is 0 or 1;
// solo: the code's solo columns.
inline GuidedTables build_guided_tables(const std::vector<uint32_t> &cols, int nwp, int R, int m,
                                        const std::vector<uint32_t> &hcol, bool binary,
                                        const SoloTable &solo) {
  GuidedTables g;
  if (!binary || R > kGuidedMaxRows || m > kGuidedMaxCols) return g;
  const int mw = (m + 31) / 32, nw = (R + 31) / 32;
  std::vector<std::vector<int>> adj(R);
  std::vector<int> cw(m, 0);
  for (int c = 0; c < m; ++c)
    for (int k = 0; k < nw; ++k)
      for (uint32_t w = cols[(size_t)c * nwp + k]; w; w &= w - 1u) {
        adj[32 * k + __builtin_ctz(w)].push_back(c);
        ++cw[c];
      }
  for (int c = 0; c < m; ++c) {
    g.max_cw = std::max(g.max_cw, cw[c]);
    if (cw[c] && !(cw[c] & 1)) g.odd = 0;
  }
  for (int r = 0; r < R; ++r) g.deg = std::max(g.deg, (int)adj[r].size());
  if (g.max_cw < 1 || g.max_cw > kGuidedMaxColWeight || g.deg > kGuidedMaxDegree) return g;
  g.gs = nw <= 4 ? 4 : 8;
  uint32_t slots = 2;
  while (slots < 2u * (uint32_t)m) slots <<= 1;
  g.tab_mask = slots - 1;
  size_t top = 0;
  auto part = [&](size_t n) {
    const size_t at = top;
    top += (n + 3) & ~(size_t)3;
    return at;
  };
  g.o_rows = part((size_t)(R + 1) * mw);
  g.o_cw = part((size_t)3 * mw);
  g.o_adj = part(((size_t)R * g.deg + 1) / 2);
  g.o_cols = part((size_t)m * g.gs);
  g.o_filt = part((size_t)1 << (kGuidedF - 5));
  g.o_tab = part((size_t)2 * slots);
  g.o_hcol = part((size_t)m);
  g.o_nib = part(nib_words(R));
  g.total = top;
  g.words.assign(top, 0u);
  uint32_t *w = g.words.data();
  std::vector<uint16_t> a((size_t)R * g.deg, (uint16_t)kNoCol);
  for (int r = 0; r < R; ++r) {
    for (size_t k = 0; k < adj[r].size(); ++k) {
      const int c = adj[r][k];
      a[(size_t)r * g.deg + k] = (uint16_t)c;
      w[g.o_rows + (size_t)r * mw + (c >> 5)] |= 1u << (c & 31);
    }
  }
  memcpy(w + g.o_adj, a.data(), sizeof(uint16_t) * a.size());
  for (uint32_t i = 0; i < slots; ++i) w[g.o_tab + 2 * i + 1] = kNoCol;
  for (int c = 0; c < m; ++c) {
    for (int b = 0; b < 3; ++b)
      if ((cw[c] >> b) & 1) w[g.o_cw + (size_t)b * mw + (c >> 5)] |= 1u << (c & 31);
    memcpy(w + g.o_cols + (size_t)c * g.gs, cols.data() + (size_t)c * nwp, sizeof(uint32_t) * nw);
    const uint32_t f = hcol[c] >> (32 - kGuidedF);
    w[g.o_filt + (f >> 5)] |= 1u << (f & 31);
    uint32_t i = hcol[c] & g.tab_mask;
    while (w[g.o_tab + 2 * i + 1] != kNoCol) i = (i + 1) & g.tab_mask;
    w[g.o_tab + 2 * i] = hcol[c];
    w[g.o_tab + 2 * i + 1] = (uint32_t)c;
  }
  memcpy(w + g.o_hcol, hcol.data(), sizeof(uint32_t) * m);
  for (int i = 0; i < nib_words(R); ++i) w[g.o_nib + i] = nib_sketch(i);
  for (size_t k = 0; k < solo.cols.size(); ++k) {
    if (solo.cols[k] < 0) continue;
    uint32_t i = solo.keys[k] & g.tab_mask;
    while (w[g.o_tab + 2 * i + 1] != (uint32_t)solo.cols[k]) i = (i + 1) & g.tab_mask;
    w[g.o_tab + 2 * i + 1] |= kSoloFlag;
  }
  return g;
}

// The descriptor's pointers into a device (or host) copy of g.words (nullptr: none).
inline void set_guided(DevCode &d, const GuidedTables &g, const uint32_t *base) {
  d.g_gs = base ? g.gs : 0;
  if (!d.g_gs) return;
  d.g_deg = g.deg;
  d.g_max_cw = g.max_cw;
  d.g_odd = g.odd;
  d.g_magic = 0xffffffffull / (unsigned)g.deg + 1ull;
  d.g_tab_mask = g.tab_mask;
  d.g_rows = base + g.o_rows;
  d.g_cw = base + g.o_cw;
  d.g_adj = reinterpret_cast<const uint16_t *>(base + g.o_adj);
  d.g_cols = base + g.o_cols;
  d.g_filt = base + g.o_filt;
  d.g_tab = base + g.o_tab;
  d.g_hcol = base + g.o_hcol;
  d.g_nib = base + g.o_nib;
  d.g_words = (int)g.total;
}

// Does every search of this code fit the chunk kernel, whatever the syndrome?  Its records
// and logicals fit a lane, weights are searched in ascending order up to wl, and the
// levels kept on the way (sets of up to wl - 2 columns, each with at most deg
// successors) fit the warp's items.  A set whose residual is zero is extended by every
// active column: for ML that happens after a match, so two levels before the last.
inline bool guided_closed(const DevCode &d) {
  if (!d.g_gs || d.n_logicos > 128) return false;
  int wl = d.Wc;
  if (d.variant == kProb) {
    wl = 5;
    for (int q = 0; q < d.n_masks; ++q)
      for (int k = 0; k < d.num_phases; ++k)
        if (d.mask_order[q][k] == 1) return false;
  }
  if (d.variant == kMl && wl > 3) return false;
  long long items = 1, level = 1;
  for (int k = 1; k <= wl - 2; ++k) {
    level *= d.g_deg;
    items += level;
    if (items > kGuidedItems) return false;
  }
  return true;
}

}  // namespace grand
