// Slab counts of the oversize tier (mg_slabs.h) under an allocator with a limit.
#include <cstdio>

#include "mg_slabs.h"

static int fails = 0;
#define CHECK(x)                                          \
  do {                                                    \
    if (!(x)) {                                           \
      std::printf("line %d: %s\n", __LINE__, #x);         \
      fails++;                                            \
    }                                                     \
  } while (0)

int main() {
  using mg::slabs_wanted;
  using mg::take_slabs;
  // a slab per waiting read, within the count, the bytes and never below what there is
  CHECK(slabs_wanted(0, 12, 64, 1 << 20, 1 << 30) == 12);
  CHECK(slabs_wanted(0, 0, 64, 1 << 20, 1 << 30) == 1);
  CHECK(slabs_wanted(0, 1000, 64, 1 << 20, 1 << 30) == 64);
  CHECK(slabs_wanted(20, 12, 64, 1 << 20, 1 << 30) == 20);
  CHECK(slabs_wanted(0, 12, 64, 256 << 20, 1 << 30) == 4);
  CHECK(slabs_wanted(3, 12, 64, 3ull << 30, 1 << 30) == 1);  // one slab larger than the limit still runs
  // memory for `room` slabs: as many as halving finds, one when there is room for one, none without
  for (int want = 1; want <= 64; want++)
    for (int room = 0; room <= 70; room++) {
      int tries = 0;
      const int got = take_slabs(want, 1, [&](int n) { return tries++, n <= room; });
      CHECK(got <= room && got <= want && (got > 0) == (room > 0) && tries <= 7);
      CHECK(room < want || got == want);
      CHECK(room >= want || 2 * got + 1 >= room || 2 * got >= want / 2);
      for (int have = 1; have < want; have++) {  // more than there are, or nothing
        const int more = take_slabs(want, have + 1, [&](int n) { return n <= room; });
        CHECK(more == 0 || (more > have && more <= room && more <= want));
        CHECK(more != 0 || room <= have);
      }
    }
  std::printf(fails ? "%d failed\n" : "ok\n", fails);
  return fails != 0;
}
