// What the attention kernels (attention.cu, attention_tile.cu) share.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "launch.h"

namespace tsr {

constexpr int kAttnMaxGroup = 8;       // heads / kv_heads <= 8
constexpr float kNullMax = -1e30f;     // running max before the first key, as the reference's kernels have it
constexpr float kLog2e = 1.4426950408889634f, kLn2 = 0.6931471805599453f;
constexpr float kNoKey = -3.0e38f;  // score of a key outside the chunk, and the running max before the first key

enum : int { kKvF32 = 0, kKvF16 = 1, kKvFp8 = 2, kKvInt8 = 3, kKvInt4 = 4 };

template <int KV>
__host__ __device__ constexpr int kv_bits() {
  return KV == kKvF32 ? 32 : KV == kKvF16 ? 16 : KV == kKvInt4 ? 4 : 8;
}

struct AttnParams {
  const float* q;
  const void* k;
  const void* v;
  const float* ks;
  const float* vs;
  // partial of (query row i, head h, chunk s) at base = (i * heads + h) * splits + s: pacc[base * head_dim ..],
  // pmax[base], psum[base]; an empty chunk is the null partial (0, kNullMax, 0)
  // (the layout of the reference's split kernels, src/backends/rocm/rocm_kernels_basic.cpp:278-330)
  float* pacc;
  float* pmax;
  float* psum;
  int m, n, heads, kv_heads, head_dim, window, causal, splits;
  unsigned long long q_base, row_base;
};

// Attention of a batch of query rows on the tensor pipe (attention_tile.cu): the whole of tsr_attention for the
// 16-bit and narrower caches, out = attention [* sigmoid(gate)].  kUnsupportedFeature: not one of its shapes.
int attention_tile(int kvkind, AttnParams p, float* out, const float* gate, cudaStream_t st);

// The same of few (row, head) pairs or keys over an FP8, int8 or 4-bit cache: asked first, kUnsupportedFeature where row
// tiles are the better choice too.
int attention_few(int kvkind, AttnParams p, float* out, const float* gate, cudaStream_t st);

}  // namespace tsr
