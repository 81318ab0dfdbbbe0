// Row cursors of a counting sort that reads its input twice: one pass counts
// a row's entries, a second one places them, taking the count down by one
// atomically per entry (`left` is the value before that).  Should the input
// change between the passes, a row sees more entries than were counted, or
// fewer; neither may reach outside the row.  Plain C++, so that the rule can
// be tested without a GPU.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define MK_ROWS_FN __host__ __device__ __forceinline__
#else
#define MK_ROWS_FN inline
#endif

namespace mk {

constexpr uint32_t kNoPlace = 0xFFFFFFFFu;

// Place of an entry in its row of `len`, or kNoPlace for one more than was
// counted.  The cursor wraps below zero there and stays wrapped, so the bound
// is tested on every entry and not only on the one that finds zero.
MK_ROWS_FN uint32_t row_place(uint32_t left, uint64_t len) {
  const uint32_t at = left - 1u;
  return at < len ? at : kNoPlace;
}

// Entries at the front of the row that nobody placed (`left` after the fill).
MK_ROWS_FN uint64_t row_gap(uint32_t left, uint64_t len) { return left <= len ? left : 0; }

}  // namespace mk
