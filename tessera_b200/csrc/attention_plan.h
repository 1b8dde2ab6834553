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

// CTAs per cluster: a power of two, one per kFewKeysPerCta keys as long as all clusters run at a time (a second wave costs
// more than twice the keys a CTA).  `resident(ctas)`: how many clusters of that size the device runs at a time, 0 where it
// does not take the size; asked only for sizes that come into question.
template <typename Resident>
inline int few_ctas(int64_t span, int64_t clusters, Resident resident, bool* one_wave) {
  int most = 1;
  while (most < kFewCluster && most * kFewKeysPerCta < span) most *= 2;
  for (int ctas = most; ctas > 0; ctas /= 2)
    if (clusters <= resident(ctas)) {
      *one_wave = true;
      return ctas;
    }
  *one_wave = false;
  return most < kFewCluster / 2 ? most : kFewCluster / 2;  // sizes every device takes
}

// Whether four rows or more are better off with the few-row kernel than with row tiles: all clusters at a time and not too
// many keys for each CTA.  Measured, FP8, few-row kernel / row tiles: 24 heads over 4 of 256, 8 rows x 512, 2048, 4096 keys 13.1 /
// 18.6, 19.5 / 25.5, 29.8 / 32.6 us; 16 x 1024 (256 keys a CTA) 19.3 / 23.9, 16 x 2048 (512) 28.3 / 28.0, 24 x 512 (256, two
// CTAs) 21.1 / 22.7, 24 x 1024 (512, two CTAs) 30.0 / 25.1, 64 x 200 (one CTA) 22.1 / 30.6, 64 x 512 32.1 / 23.6; 16 heads over 2 of
// 128, 32 x 4096 (1024) 22.8 / 28.8, 48 x 2048 (1024, two CTAs) 23.4 / 24.1, 128 x 512 (one CTA) 17.0 / 17.2.
inline bool few_rows_win(int64_t span, int ctas, bool one_wave, int head_dim) {
  return one_wave && span * head_dim <= static_cast<int64_t>(ctas) * (ctas >= 4 ? 512 : 256) * 256;
}

// The least products (of one of the two contractions) that pay for row tiles where the chunk kernel is the other choice.
// fp16 cache (three products a tile), row tiles / chunk kernel, 24 heads over 4 of 256: 16 rows x 200 keys (2.0e7) 24.1 / 20.1 us,
// 24 x 200 (2.9e7) 24.9 / 22.2, 64 x 64 (2.5e7) 28.8 / 30.4, 32 x 200 (3.9e7) 25.2 / 31.3; 8 x 512 (2.5e7) 20.0 / 16.7, 12 x 512
// (3.8e7) 24.2 / 24.4, 4 x 2048 (5.0e7) 26.4 / 26.9; 16 heads over 2 of 128: 24 x 512 (2.5e7) 18.2 / 20.3, 8 x 2048 (3.4e7) 21.5 / 20.6,
// 12 x 2048 (5.0e7) 23.9 / 28.7.  What the narrower caches bring here is not one wave of the few-row kernel: FP8, 24 x 64 (9.4e6)
// 20.0 / 17.2, 32 x 64 (1.3e7) 20.0 / 19.4, 48 x 64 21.1 / 26.4.
inline double tile_least(bool f16, int64_t m) { return !f16 ? 1.2e7 : m >= 16 ? 2.2e7 : 4.5e7; }

}  // namespace tsr
