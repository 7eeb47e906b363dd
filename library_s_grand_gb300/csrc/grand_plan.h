// grand_plan.h -- what the host decides about a batch's launches (no CUDA calls).
#pragma once

#include <algorithm>
#include <vector>

#include "grand_common.h"
#include "grand_guided_tables.h"

namespace grand {

// Which kernels decode the batch, and its chunks: b.has_ml, b.guided, b.chunk, b.fast, from its
// codes, b.num_shots and b.shot_map.  fast: the chunk step may be used (GRAND_FAST).
inline void plan_batch(DevBatch &b, const DevCode *codes, int ncodes, int sm_count, bool fast) {
  bool any = false, all = true;
  long long entries = 1;  // int32 entries of the longest record that the chunk step takes
  b.has_ml = 0;
  for (int i = 0; i < ncodes; ++i) {
    b.has_ml |= codes[i].variant == kMl;
    any = any || codes[i].g_gs;
    all = all && guided_closed(codes[i]);
    if (!codes[i].packed && chunk_takes(codes[i])) entries = std::max<long long>(entries, codes[i].rec_len);
  }
  all = all && entries <= 32 * kFastBallots && !b.shot_map;
  b.guided = !fast || !any ? kGuidedNone : (all ? kGuidedAll : kGuidedFirst);
  // Back-to-back records of a whole chunk fit its ballot area: past it every shot of the chunk
  // takes the per-shot path (100000 errors of a 60 x 300 code without tables 300 us in these
  // chunks; 20000 of them 93, and 159 in chunks of 32).
  const int most = (int)std::max<long long>(std::min<long long>(kMaxChunk, 32 * kFastBallots / entries), 1);
  // Full waves of the resident warps, in chunks as large as they may be: a chunk costs its
  // records' round trips whatever its size, a part wave costs a whole one (twice the chunks
  // in half the size: headline 30.8 -> 40.3 us, noisy [[288]] 52 -> 62).  The decode kernel's
  // warps draw chunks, so there only a batch of less than a wave is split further (256 errors
  // of the 60 x 300 code 47 us, 57 in chunks of 27).
  const int warps = sm_count * kChunkMinBlocks * kChunkWarps;
  const int waves = b.guided ? (b.num_shots - 1) / (warps * most) + 1 : 1;
  b.chunk = std::min((b.num_shots - 1) / (warps * waves) + 1, most);
  // A warp for every shot: straight to the per-shot path, which reads the record once (256 errors
  // of the 60 x 300 code 39 us, 46 through the chunk step).
  b.fast = fast && (b.guided || b.num_shots > warps);
  if (b.guided == kGuidedAll) b.deferred = nullptr;  // nothing is ever deferred
}

// The return code for the status bits of a finished batch (those of a full job table or arena
// apart): a warp that gave up waiting left shots undecoded, which comes before a set that
// was too large, reported in its result.
inline int status_code(unsigned status) {
  if (status & (kStatusCasLimit | kStatusWaitLimit)) return GRAND_ERR_CUDA;
  return status & kStatusTamLimit ? GRAND_ERR_LIMIT : 0;
}

// The shots of the next round after one in which some found the job table or the arena full:
// those of map (in the first round: of all shots) whose re-run flag is set.  False when there
// are as many as before, so that a further round would leave the same ones: each of them
// alone needs more than there is.
inline bool next_round(std::vector<int> &map, const std::vector<int> &flags, bool first) {
  const size_t before = first ? flags.size() : map.size();
  std::vector<int> next;
  if (first) {
    for (size_t i = 0; i < flags.size(); ++i)
      if (flags[i]) next.push_back((int)i);
  } else {
    for (int i : map)
      if (flags[i]) next.push_back(i);
  }
  map.swap(next);
  return map.size() < before;
}

}  // namespace grand
