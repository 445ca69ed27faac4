// How many workspaces (slabs) the oversize tier of a classification call gets.
#pragma once
#include <algorithm>
#include <cstdint>

namespace mg {

// A slab for each waiting read (and no fewer than there are), within `most` and `most_bytes` in all;
// one at least.
inline int slabs_wanted(int have, uint32_t waiting, int most, uint64_t bytes, uint64_t most_bytes) {
  const uint64_t fit = std::max<uint64_t>(1, most_bytes / std::max<uint64_t>(1, bytes));
  const uint64_t want = std::max<uint64_t>({1, (uint64_t)std::max(0, have), waiting});
  return (int)std::min<uint64_t>(std::min<uint64_t>(want, (uint64_t)most), fit);
}

// The slabs that memory allows: get(n) tries to allocate n; want, then half as many each time, the
// last time `least`. 0: not even that. Fewer slabs than reads only cost time (the tier's blocks take
// the reads in turn), so the device being short of memory is no error while one slab fits.
template <class Get>
int take_slabs(int want, int least, Get&& get) {
  for (int n = want; n >= least && n > 0; n = n > least ? std::max(least, n / 2) : 0)
    if (get(n)) return n;
  return 0;
}

}  // namespace mg
