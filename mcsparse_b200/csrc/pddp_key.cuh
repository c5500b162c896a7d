// Sort keys of the query grouping (pddp.cu): the order-preserving image of a row's projection above the row's position inside
// its node.  Positions make the keys unique, so the sort is stable by construction.
#pragma once
#include <cstdint>

#ifdef __CUDACC__
#define MCS_KEY_FN __host__ __device__ inline
#else
#define MCS_KEY_FN inline
#endif

namespace mcs {

constexpr unsigned long long kPadKey = 0xFFFFFFFFFFFFFFFFull;     // slots beyond a node: behind every row

MCS_KEY_FN unsigned long long sort_key(uint32_t projection_key, int position) {
  return (static_cast<unsigned long long>(projection_key) << 32) | static_cast<uint32_t>(position);
}

// Position that a sorted key names, inside a node of `size` rows whatever the key holds: the sorts are queued before it is known
// whether a wait of the kernel in front of them expires, and what they read back is used as a row number by everything that follows.
MCS_KEY_FN int key_position(unsigned long long key, int size) {
  const uint32_t position = static_cast<uint32_t>(key), last = static_cast<uint32_t>(size - 1);
  return static_cast<int>(position < last ? position : last);
}

}  // namespace mcs
