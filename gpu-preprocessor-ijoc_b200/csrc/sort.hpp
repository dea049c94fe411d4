// Device sort primitive shared by the duplicate-detection rules.
#pragma once

#include "common.cuh"

namespace gpp {
// Bits that the values 0 .. top can have set.
inline uint64_t bits_up_to(int64_t top) {
  return top <= 0 ? 0 : ~uint64_t(0) >> __builtin_clzll(uint64_t(top));
}
// Stable sort of n (key, value) pairs by key, in place.  `may_vary` names the
// key bits to sort by: those that can differ between keys, or only the upper
// ones of them when the input is already in order by the lower ones.  `ask`, for a
// caller that waits for the sort anyway and knows nothing of the keys: the host waits for
// the digit counts and leaves out the passes of constant digits.
void radix_sort_pairs(uint64_t* keys, int32_t* vals, int64_t n, cudaStream_t s, uint64_t may_vary = ~uint64_t(0),
                      bool ask = false);
// Test hook: the polls after which a look-back gives up (<= 0 for the default).
void inject_sort_wait_limit(int polls);
// The same sort with its scratch in a fixed device array (no allocation);
// n is at most GPP_SORT_STATIC_MAX_PAIRS.
void radix_sort_pairs_static(uint64_t* keys, int32_t* vals, int64_t n, cudaStream_t s);
}  // namespace gpp
