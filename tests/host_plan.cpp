// Host-side checks of what the library decides before a launch, for
// tests/test_plan_host.py.
//
// Usage: host_plan layout | rounds | status
#include <cstdio>
#include <cstring>
#include <vector>

#include "grand_host.h"
#include "grand_plan.h"

using namespace grand;

// The per-shot buffer's parts for every batch that fits one allocation: inside it, apart,
// aligned, and in the same places whatever the batch's size (an entry of a later launch must
// not lie where an earlier one left flags or records).
static int layout() {
  for (size_t most : {1u, 2u, 3u, 7u, 32u, 33u, 1000u, 4097u, 65536u, 1000003u}) {
    const size_t bytes = shot_buffer_bytes(most);
    if (shot_capacity(bytes) != most) return 1;
    char *base = reinterpret_cast<char *>(size_t{1} << 20);
    const char *queue = reinterpret_cast<char *>(shot_queue(base, bytes));
    const char *cache = reinterpret_cast<char *>(shot_rec_cache(base, bytes));
    if ((queue - base) % 8 || (cache - base) % 16) return 2;
    for (size_t n = 1; n <= most; n = n < most && 2 * n > most ? most : 2 * n) {
      if (shot_buffer_bytes(n) > bytes) return 3;
      if (base + sizeof(int) * n > queue || queue + 8 * n > cache) return 4;
      if (cache + sizeof(uint32_t) * kRecCacheWords * n > base + bytes) return 5;
    }
  }
  return 0;
}

// Rounds of a batch against an arena that `fit` shots fill: each shot is searched once, in
// however many rounds that takes, and shots that alone outgrow it are told from the rest.
static int rounds() {
  for (int shots : {1, 63, 1000}) {
    for (int fit : {1, 7, 2000}) {
      for (int huge : {0, 1, 5}) {
        std::vector<int> flags(shots, 0), searched(shots, 0), map;
        int round = 0;
        for (;; ++round) {
          if (round > shots + 1) return 1;
          int room = fit, any = 0;
          const int todo = round ? (int)map.size() : shots;
          for (int k = 0; k < todo; ++k) {
            const int i = round ? map[k] : k;
            const bool full = i % 97 < huge || room == 0;
            flags[i] = full;
            any |= full;
            if (!full) --room, ++searched[i];
          }
          if (!any) {
            map.clear();
            break;
          }
          const bool fewer = next_round(map, flags, round == 0);
          if (map.empty() || !fewer) break;
        }
        std::vector<int> left(shots, 0);
        for (int i : map) left[i] = 1;
        for (int i = 0; i < shots; ++i)
          if (searched[i] != (i % 97 < huge ? 0 : 1) || left[i] != (i % 97 < huge ? 1 : 0)) return 2;
      }
    }
  }
  return 0;
}

// Every combination of status bits: a wait or retry that gave up is an error whatever else
// was raised.
static int status() {
  for (unsigned st = 0; st < 64; ++st) {
    const bool gave_up = st & (kStatusCasLimit | kStatusWaitLimit);
    const int want = gave_up ? GRAND_ERR_CUDA : (st & kStatusTamLimit ? GRAND_ERR_LIMIT : 0);
    if (status_code(st) != want) return 1;
  }
  return 0;
}

int main(int argc, char **argv) {
  if (argc == 2 && !strcmp(argv[1], "layout")) return layout();
  if (argc == 2 && !strcmp(argv[1], "rounds")) return rounds();
  if (argc == 2 && !strcmp(argv[1], "status")) return status();
  return 9;
}
