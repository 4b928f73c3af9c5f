// C entry for tests/test_lookback.py: items_before with words that are published
// only after a number of looks, or never.
#include "lookback.h"

// kind[t]: 0 never published, 1 the tile's own count, 2 the count of all tiles up
// to it; after[t]: looks at tile t that find nothing; counted[t] += 1 where the
// tile's items are counted; looked: words read. Reads outside [0, tile) are
// reported as ~0.
extern "C" uint32_t lookback(int64_t tile, uint32_t limit, const uint32_t *count, const uint8_t *kind, uint32_t *after,
                             uint32_t *counted, uint64_t *looked) {
  bool out = false;
  uint32_t r = tpm::items_before(
      tile, limit,
      [&](int64_t t) -> uint32_t {
        ++*looked;
        if (t < 0 || t >= tile) {
          out = true;
          return tpm::kAll;
        }
        if (after[t]) {
          after[t]--;
          return 0u;
        }
        if (kind[t] == 0) return 0u;
        uint32_t v = count[t];
        if (kind[t] == 2)
          for (int64_t q = 0; q < t; q++) v += count[q];
        return v | (kind[t] == 2 ? tpm::kAll : tpm::kOwn);
      },
      [&](int64_t t) -> uint32_t {
        if (t < 0 || t >= tile) {
          out = true;
          return 0u;
        }
        counted[t]++;
        return count[t];
      });
  return out ? 0xffffffffu : r;
}
