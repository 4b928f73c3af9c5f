// The look-back of a single-sweep radix pass (sort.cu): a tile learns how many
// items of a digit lie in the tiles before it from the words that those publish
// (Merrill and Garland, "Single-pass Parallel Prefix Scan with Decoupled
// Look-back", 2016). Plain C++ over the two ways to a tile's count, so that it
// runs on the host too.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define TPM_LOOK __host__ __device__ __forceinline__
#else
#define TPM_LOOK inline
#endif

namespace tpm {

// A tile's word per digit: its own count (kOwn) or that of all tiles up to and
// with it (kAll); 0 until it is published.
constexpr uint32_t kOwn = 1u << 30, kAll = 2u << 30, kCount = kOwn - 1u;

// The digit's items in the tiles before `tile`, looked up four tiles at a time.
// word(t): tile t's word now; count(t): the digit's items in tile t, counted
// from the items themselves, which the pass does not change. After `limit` looks
// in all, tiles whose word is missing are counted, so the look-back ends with the
// right number whatever the other tiles do.
template <class Word, class Count>
TPM_LOOK uint32_t items_before(int64_t tile, uint32_t limit, Word word, Count count) {
  uint32_t before = 0, looks = 0;
  int64_t t = tile - 1;
  while (t >= 0) {
    uint32_t s[4];
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int q = 0; q < 4; q++) s[q] = t - q >= 0 ? word(t - q) : kAll;
    bool done = false;
#ifdef __CUDACC__
#pragma unroll
#endif
    for (int q = 0; q < 4; q++) {
      if (done || s[q] < kOwn) break;
      before += s[q] & kCount;
      t--;
      done = s[q] >= kAll;
    }
    if (done) break;
    if (++looks > limit && t >= 0) before += count(t--);
  }
  return before;
}

}  // namespace tpm
