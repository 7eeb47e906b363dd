// grand_plan.h -- what the host decides about a batch's launches (no CUDA calls).
#pragma once

#include <vector>

namespace grand {

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
