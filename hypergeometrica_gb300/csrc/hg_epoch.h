// hg_epoch.h -- the epochs that tell one run's carry flags from another's.
#pragma once

#include <cstdint>

namespace hg {

// A tile's published aggregate carries the epoch of its run, so that a word an
// earlier run left there is not taken for this one's.  The persistent schedule
// clears its flags before every run and always has the first.
constexpr uint32_t kPersistEpoch = 1;

// Epochs of the runs that share one flag array (zeroed once, when allocated):
// another one for each run, never 0 or kPersistEpoch.
struct ScanEpoch {
  uint32_t last = kPersistEpoch;
  uint32_t next() {
    last = last == UINT32_MAX ? kPersistEpoch + 1 : last + 1;
    return last;
  }
};

}  // namespace hg
