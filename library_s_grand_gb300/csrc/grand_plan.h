// grand_plan.h -- what the host decides about a batch's launches (no CUDA calls).
#pragma once

#include <vector>

#include "grand_common.h"

namespace grand {

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
