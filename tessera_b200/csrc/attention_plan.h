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

constexpr int kFewCluster = 16;  // CTAs of a cluster of the few-row kernel at most
// Keys in each CTA before another CTA joins.  A CTA takes 128 keys a trip, but what a short call spends is the loads'
// latency and the cluster's merge, which more CTAs share: one row of 24 heads over 4 of 256, 128 / 256 / 512 keys, 16 keys a
// CTA 7.5 / 7.8 / 7.9 us, 64 keys 9.1 / 8.3 / 7.7, 128 keys 12.6 / 10.1 / 9.0; from 1024 keys on all the same.
constexpr int kFewKeysPerCta = 16;

}  // namespace tsr
