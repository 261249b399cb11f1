// One row per request (a decoding step): which keys a part of a row's work takes, for the kernel that writes work lists and for those that need none.
#pragma once
#include <stdint.h>

namespace omc {

struct LatentDecodeRows {
  const int32_t* pos;   // of every row
  const int32_t* slot;
  int parts;            // ranges of its keys
};

// Keys [from, to) of range i: a row at position pos sees the last min(pos + 1, window) keys, cut into `parts` ranges of whole tiles of 64 (those past the end are empty)
__device__ __forceinline__ void latent_decode_range(int pos, int window, int parts, int i, int& from, int& to) {
  const int keys = pos + 1, low = max(0, keys - window);
  const int span = ((keys - low + parts - 1) / parts + 63) / 64 * 64;
  from = min(low + i * span, keys), to = min(low + (i + 1) * span, keys);
}

}  // namespace omc
