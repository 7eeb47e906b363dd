// Host-side checks of what the library decides before a launch, for
// tests/test_plan_host.py.
//
// Usage: host_plan layout
#include <cstdio>
#include <cstring>
#include <vector>

#include "grand_host.h"

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

int main(int argc, char **argv) {
  if (argc == 2 && !strcmp(argv[1], "layout")) return layout();
  return 9;
}
