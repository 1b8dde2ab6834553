// How attention_tile.cu cuts its work: host arithmetic only.
#pragma once

#include <stdint.h>

namespace tsr {

constexpr int kTileRows = 128, kTileKeys = 64;  // (row, head) pairs of a row tile, keys of a step

// The most keys a row tile walks over: from the window of its first row to the position of its last.
inline int64_t tile_span(int64_t m, int64_t n, uint64_t q_base, int64_t window, bool causal, int64_t group) {
  int64_t span = n;
  if (causal && window != 0 && window + kTileRows / group + 1 < span) span = window + kTileRows / group + 1;
  if (causal && q_base + static_cast<uint64_t>(m) < static_cast<uint64_t>(span)) span = static_cast<int64_t>(q_base) + m;
  return span;
}

}  // namespace tsr
