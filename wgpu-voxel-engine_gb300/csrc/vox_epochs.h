// vox_epochs.h — when look-back words have to be zeroed (host).
//
// The words of a look-back carry the low 24 bits of their launch's epoch. A launch advances the
// epoch by one (one that timed out by at most two), so words that were written 2^24 epochs ago
// would pass for published ones. They are zeroed well before: at the first launch that uses them
// with kStateWipePeriod or more launches behind the last zeroing. The count is compared, not
// tested for a multiple: launches that use other words (a graph's replays) advance it too, and
// would step over the multiples.
// Plain C++, so that host tests check the rule itself.
#pragma once

namespace vox {

constexpr unsigned long long kStateWipePeriod = 1ull << 22;

struct EpochWipe {
  unsigned long long wiped_at = 0;  // launches before the words were last zeroed
  // Whether the words have to be zeroed ahead of a launch with `launches` launches before it
  // (the caller then does so).
  bool due(unsigned long long launches) {
    if (launches - wiped_at < kStateWipePeriod) return false;
    wiped_at = launches;
    return true;
  }
};

}  // namespace vox
