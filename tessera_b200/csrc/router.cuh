// Device pieces of the expert router: the top_k of a row of logits and the gates (top_k_rows: forward_elementwise.cu,
// moe_gate and the two merged: moe.cu).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "codec.cuh"

namespace tsr {

constexpr int kRouterThreads = 256;
struct TopKShared {
  float bv[8];
  uint32_t bi[8];
  uint32_t taken[32];
  float row[1024];   // top_k_small: the row
  float chosen[32];  // and its values, for the gates of a merged launch
};

// One row by a CTA of kRouterThreads: top_k rounds of a block-wide arg-max over the values not taken yet; among equal
// values the lowest index wins.
__device__ inline void top_k_block(const float* row, uint32_t* ids, float* vals, size_t vocab, int top_k, TopKShared& shared) {
  for (int p = 0; p < top_k; ++p) {
    float best = -INFINITY;
    uint32_t arg = 0xFFFFFFFFu;
    for (size_t c = threadIdx.x; c < vocab; c += blockDim.x) {
      const float x = row[c];
      bool used = false;
      for (int t = 0; t < p; ++t) used = used || shared.taken[t] == static_cast<uint32_t>(c);
      if (!used && (x > best || (x == best && static_cast<uint32_t>(c) < arg) || arg == 0xFFFFFFFFu)) {
        best = x;
        arg = static_cast<uint32_t>(c);
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xFFFFFFFFu, best, o);
      const uint32_t oi = __shfl_xor_sync(0xFFFFFFFFu, arg, o);
      if (oi != 0xFFFFFFFFu && (arg == 0xFFFFFFFFu || ov > best || (ov == best && oi < arg))) {
        best = ov;
        arg = oi;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      shared.bv[threadIdx.x >> 5] = best;
      shared.bi[threadIdx.x >> 5] = arg;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int x = 1; x < 8; ++x)
        if (shared.bi[x] != 0xFFFFFFFFu && (shared.bi[0] == 0xFFFFFFFFu || shared.bv[x] > shared.bv[0] || (shared.bv[x] == shared.bv[0] && shared.bi[x] < shared.bi[0]))) {
          shared.bv[0] = shared.bv[x];
          shared.bi[0] = shared.bi[x];
        }
      shared.taken[p] = shared.bi[0];
      vals[p] = shared.bi[0] == 0xFFFFFFFFu ? -INFINITY : shared.bv[0];
      ids[p] = shared.bi[0] == 0xFFFFFFFFu ? 0u : shared.bi[0];
    }
    __syncthreads();
  }
}

// The same for rows of up to 32 P logits (a router's; P up to 32): warp 0 has the row in registers (lane l columns
// l, l + 32, ...) and keeps each lane's largest; a round is a warp-wide arg-max and a rescan in the winner's lane, without
// a barrier.  256 experts, eight selected: with moe_gate in one launch 7.3 us, the two launches before took 9.6
// and 7.6.  A row with a NaN takes the rounds above, whose order of comparisons decides there.
constexpr uint64_t kTopKSmall = 1024;
template <int P, typename Between>
__device__ __forceinline__ void top_k_small(const float* __restrict__ row, uint32_t* ids, float* vals, int vocab, int top_k,
                                            TopKShared& shared, Between between) {
  constexpr int kPer = (P * 32 + kRouterThreads - 1) / kRouterThreads;
  float x[kPer];
  bool nan = false;
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int c = threadIdx.x + i * kRouterThreads;
    x[i] = c < vocab ? row[c] : 0.0f;
  }
  between();  // what the caller does while the row is on its way
#pragma unroll
  for (int i = 0; i < kPer; ++i) {
    const int c = threadIdx.x + i * kRouterThreads;
    nan |= x[i] != x[i];
    if (c < vocab) shared.row[c] = x[i];
  }
  if (__syncthreads_or(nan)) {
    top_k_block(row, ids, vals, vocab, top_k, shared);
    if (threadIdx.x < top_k) shared.chosen[threadIdx.x] = vals[threadIdx.x];
    return;
  }
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  float v[P];
  uint32_t taken = 0;  // bit i: column lane + 32 i is out (or beyond the row)
#pragma unroll
  for (int i = 0; i < P; ++i) {
    const bool in = lane + i * 32 < vocab;
    v[i] = in ? shared.row[lane + i * 32] : 0.0f;
    if (!in) taken |= 1u << i;
  }
  float best;
  uint32_t arg;
  auto scan = [&] {
    best = -INFINITY, arg = 0xFFFFFFFFu;
#pragma unroll
    for (int i = 0; i < P; ++i)
      if (!(taken >> i & 1u) && (arg == 0xFFFFFFFFu || v[i] > best)) best = v[i], arg = lane + i * 32;
  };
  scan();
  for (int p = 0; p < top_k; ++p) {
    float b = best;
    uint32_t a = arg;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float ov = __shfl_xor_sync(0xFFFFFFFFu, b, o);
      const uint32_t oi = __shfl_xor_sync(0xFFFFFFFFu, a, o);
      if (oi != 0xFFFFFFFFu && (a == 0xFFFFFFFFu || ov > b || (ov == b && oi < a))) b = ov, a = oi;
    }
    if (lane == 0) {
      const float value = a == 0xFFFFFFFFu ? -INFINITY : b;
      vals[p] = value;
      shared.chosen[p] = value;
      ids[p] = a == 0xFFFFFFFFu ? 0u : a;
    }
    if (a != 0xFFFFFFFFu && (a & 31u) == static_cast<uint32_t>(lane)) {
      taken |= 1u << (a >> 5);
      scan();
    }
  }
}

// moe_gate in two halves: the partial sums of x . w (one per warp in `red`; a barrier before the second half), then by
// warp 0 the softmax over the top_k selected logits (a logit a lane, the exponentials added in slot order) and the
// sigmoid.  One thread doing the second half took 7.6 us, most of them serial exponentials.
__device__ __forceinline__ void moe_gate_dot(const float* __restrict__ x, const float* __restrict__ w, int hidden, float* red) {
  float dot = 0.0f;
#pragma unroll 8
  for (int t = threadIdx.x; t < hidden; t += kRouterThreads) dot = fmaf(x[t], w[t], dot);
  dot = warp_sum(dot);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = dot;
}
__device__ __forceinline__ void moe_gate_finish(const float* vals, float* wts, float* sig, int top_k, const float* red) {
  if (threadIdx.x >= 32) return;
  const int lane = threadIdx.x;
  float m = -3.402823466e+38f;
  for (int p = lane; p < top_k; p += 32) m = fmaxf(m, vals[p]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, o));
  float sum = 0.0f;
  for (int p0 = 0; p0 < top_k; p0 += 32) {
    const float e = p0 + lane < top_k ? expf(vals[p0 + lane] - m) : 0.0f;
    for (int p = 0; p < 32 && p0 + p < top_k; ++p) sum += __shfl_sync(0xFFFFFFFFu, e, p);
  }
  for (int p = lane; p < top_k; p += 32) wts[p] = expf(vals[p] - m) / sum;
  if (lane == 0) {
    float total = 0.0f;
    for (int i = 0; i < kRouterThreads / 32; ++i) total += red[i];
    sig[0] = 1.0f / (1.0f + expf(-total));
  }
}

}  // namespace tsr
