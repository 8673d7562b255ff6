// Launch shape of batches without a tuned one; plain C++, so that the rule is tested on the CPU too.
#pragma once
#include <algorithm>
#include <cstdint>

namespace pxl {

// Blocks per event: enough for eight waves of eight blocks per SM, at most 256, and at least one per 1024 words of
// the batch's mean event, between 4 and 32. Events differ in size and the blocks of one share its work, so a
// batch cut to one wave (1184 / E blocks, at least 4) waits for its largest events: 111 events of pileup 1 to
// 200 13.2 ms, with 85 blocks 9.3; 24 of them 3.9 and, with 256, 3.7; 512 of pileup 1 to 100 13.6 ms with 4 blocks,
// 11.5 with the 18 of eight waves, 11.3 with 32. Of equal events, whose blocks only become shorter: 512 of pileup
// 50 10.2 ms with 4, 9.5 with 18 or 32. Twice as many as eight waves: 9.1 ms (111 uneven), but 3.36 instead of
// 3.28 ms for 111 equal ones. Small events fill few blocks, and the empty ones are launched all the same: 4096
// events of 10 tracks 1.52 ms with 4 blocks, 2.55 with 32, of 100 tracks 3.85 and 4.93; 2048 of pileup 10 9.8 with 4,
// 10.2 with 10, 10.5 with 32. The words of a batch on the device are not known (0): it gets the eight waves alone.
inline int blocks_per_event(int events, uint64_t batch_words) {
  const int n = std::max(1, events);
  const uint64_t words = batch_words / uint64_t(n);
  const int least = std::max(4, int(std::min<uint64_t>(32, words / 1024)));
  return std::max(least, std::min(256, 148 * 64 / n));
}

}  // namespace pxl
