// Output slots of a single dilation (dilate_fast): `cap` intervals for every
// column, then a spill region for the columns with more; and the largest input of patches. Host only.
#pragma once
#include <stdint.h>

#include <algorithm>

namespace vo {

struct SlotLayout {
  int cap = 1;
  int64_t spill = 0;
};

constexpr int64_t kSlotSpare = 4096;         // spill space beyond what is asked for
constexpr int64_t kSlotMost = 4294967295LL;  // slot indices are unsigned 32-bit: columns and spill together
constexpr int64_t kSegmentsMost = 2147483647LL;  // a result of more segments is refused

// Inputs of up to so many segments (or slots) may go by patches, whose entries hold the index of a value, two per segment,
// in a signed 32-bit integer; larger ones go by columns.
constexpr int64_t kPatchSegments = 1LL << 30;

// At first: from the input's mean segment count per column, with an eighth of the columns' slots to spill.
inline SlotLayout slots_first(int64_t ncols, double mean_segs) {
  SlotLayout s;
  s.cap = mean_segs > 24.0 ? 64 : mean_segs > 10.0 ? 48 : mean_segs > 6.0 ? 32 : 24;
  s.cap = (int)std::max<int64_t>(1, std::min<int64_t>(s.cap, kSlotMost / 9 * 8 / std::max<int64_t>(ncols, 1)));
  s.spill = std::max<int64_t>(kSlotSpare, ncols * s.cap / 8);
  return s;
}

// For a run most of whose columns have unions beyond the first tiers' lists: slots for 128 intervals each and as many
// again to spill, up to 4 GB of either.
inline void slots_many(int64_t ncols, SlotLayout &s) {
  const int64_t n = std::max<int64_t>(ncols, 1);
  s.cap = (int)std::max<int64_t>(s.cap, std::min<int64_t>(128, (1LL << 28) / n));
  s.spill = std::max<int64_t>(s.spill, std::min<int64_t>(n * s.cap, std::min<int64_t>(1LL << 28, kSlotMost - n * s.cap)));
}

// After a run whose columns asked for `need` intervals of spill space, more than there was. Where that and
// the columns' slots together pass the slot range, the slots shrink until any result that is not refused
// fits: with it all in the spill region. False when the result is refused.
inline bool slots_next(int64_t ncols, int64_t need, SlotLayout &s) {
  if (need > kSegmentsMost) return false;
  s.spill = need + kSlotSpare;
  if (ncols * s.cap + s.spill > kSlotMost) {
    s.spill = kSegmentsMost + kSlotSpare;
    s.cap = (int)((kSlotMost - s.spill) / std::max<int64_t>(ncols, 1));
  }
  return s.cap >= 1;
}

}  // namespace vo
