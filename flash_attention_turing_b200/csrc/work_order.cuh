// The order in which the persistent kernels take the work items of a causal batch: heaviest first over a whole SECTION of heads, then
// the next section.  An item can be a tenth of a launch.  Head by head (heaviest first within each) the heaviest item of the last
// head is begun when the rest is nearly over, and its SM runs on alone.  A section ends with the lightest items of all its heads
// instead, and the next section's heavy ones start under them.  It is no larger than what the L2 cache holds of the rows that the
// items stream, so that these are still read from memory once.
// Head by head against this (us): forward B2 S2047 Hq16 Hkv4 D128 58.1 -> 42.9, B1 S3001 Hq32 Hkv8 100.9 -> 82.3, B4 S4096 H32 639 -> 590,
// B16 S1024 223 -> 205, 8 packed documents of 256-4096 tokens H16 133 -> 114; backward (dK/dV starts on what dQ leaves idle, so it had
// less to lose) B1 S3001 314 -> 283, B2 S2047 176 -> 172.  Sections of 16 and 64 MB: the same within the spread.
#pragma once

#include <stdint.h>

namespace fa {

// Bytes of streamed rows (K and V; for dK/dV Q and dO) per section: well below the 126 MB of L2, half of which is each die's.
constexpr int64_t kSectionBytes = 32 << 20;

// Host: rows of `row_bytes` that a section may hold; 0, a head (or group) per section, where the order gains nothing because all items of a
// head are equal or nearly so: no causal mask, or few queries at the end of many keys.  The heads of a group are then taken tile by tile; one
// head after the other took the same, 17 grouped shapes without mask 0.98-1.02.
inline int section_rows(bool causal, int seqlen_q, int seqlen_k, int64_t row_bytes) {
  return causal && 4 * static_cast<int64_t>(seqlen_q) >= seqlen_k ? static_cast<int>(kSectionBytes / row_bytes) : 0;
}

#ifdef __CUDACC__
struct HeadPlace {
  int head, place;  // place: position among the items of the head, 0 = heaviest
};
// Item r of `heads` heads with `count` items each, in units of `unit` heads that share their streamed rows (of which there are `rows`).
__device__ __forceinline__ HeadPlace section_item(int r, int heads, int count, int unit, int rows, int rows_per_section) {
  if (rows_per_section == 0) {
    const int group = r / (unit * count), rest = r - group * unit * count, place = unit == 1 ? rest : rest / unit;
    return {group * unit + rest - place * unit, place};
  }
  if (static_cast<int64_t>(rows) * heads <= static_cast<int64_t>(rows_per_section) * unit) {  // one section: a division, not four (64 packed texts 103 -> 100 us)
    const int place = r / heads;
    return {r - place * heads, place};
  }
  const int section = min(heads / unit, max(1, rows_per_section / max(rows, 1))) * unit;
  const int first = r / (section * count) * section;
  const int rest = r - first * count, n = min(section, heads - first);
  return {first + rest % n, rest / n};
}
#endif

}  // namespace fa
