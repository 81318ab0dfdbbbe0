// Places the entries of a fill pass by the row cursors of mk_rows.h after a
// count pass that saw other entries: argv = counted and filled entries of
// each row, in pairs.  Exits 1 when a place lies outside its row or is taken
// twice, or when the gap is not exactly the places left open.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "mk_rows.h"

int main(int argc, char **argv) {
  for (int r = 1; r + 1 < argc; r += 2) {
    const uint32_t len = (uint32_t)std::strtoul(argv[r], nullptr, 10);
    const uint32_t fill = (uint32_t)std::strtoul(argv[r + 1], nullptr, 10);
    uint32_t cursor = len, placed = 0;
    std::vector<char> row(len, 0);
    for (uint32_t e = 0; e < fill; ++e) {
      const uint32_t at = mk::row_place(cursor--, len);  // atomicSub: the value before
      if (at == mk::kNoPlace) continue;
      if (at >= len || row[at]++) {
        std::printf("row of %u, %u filled: entry %u at %u\n", len, fill, e, at);
        return 1;
      }
      ++placed;
    }
    const uint64_t gap = mk::row_gap(cursor, len);
    if (gap + placed != len) return 1;
    for (uint64_t j = 0; j < len; ++j)
      if ((row[j] == 0) != (j < gap)) return 1;
  }
  return 0;
}
