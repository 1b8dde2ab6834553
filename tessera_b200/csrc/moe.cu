// Routed-expert kernels of a mixture-of-experts layer for one token: the expert
// ids live in device memory, so the launch gathers the rows of the selected
// experts out of the whole 3-D expert tensors.  Contracts:
// src/backends/rocm/rocm_kernels.hpp:604-640 of the reference (moe_gate,
// moe_scale_add, moe_experts_gate_up_q4k, moe_experts_down_q4k / _q6k); the
// arithmetic of a row is the reference's block dot
// (src/core/numerics/gemm.cpp:18-41,88-99), re-associated per sub-block as in
// the warp-per-row family (gemv_rows.cu).
//
// Gathers: top_k experts x inter rows x (gate + up) and top_k x
// hidden rows per token (9.4 MB + 4.7 MB per layer), every weight
// byte read once with 16-byte loads, asked for before the activations are staged in
// shared memory.  Bound: latency (ids, then rows all over the tensors) and the dot products; 256 experts of
// 2048 -> 512 -> 2048, eight selected: gate/up 12.8 -> 10.3 us, down 10.0 -> 7.3 us with the activations
// laid out for the eight lanes of a block (four-way bank conflicts before) and the loads in front.
#include "codec.cuh"
#include "launch.h"
#include "router.cuh"
#include "tessera_b200.h"

namespace tsr {

namespace {

constexpr int kMoeWarps = 8;

// Activations in shared memory as q4k_chunk_dot reads them: of each block of 256, quad v (0..3) of the sixteen elements
// that chunk c8's low (side 0) or high (side 1) nibbles multiply lies at quad (2 v + side) * 8 + c8.  Eight lanes of
// eight chunks then read 128 consecutive bytes; in element order they met on two of the banks' eight quads, and those
// conflicts bound the kernel.  `count` floats (a multiple of 256) from global memory.
__device__ __forceinline__ void stage_activations(float* xs, const float* __restrict__ src, int count) {
  for (int t = threadIdx.x; t < count / 4; t += blockDim.x) {
    const int v = t & 3, group = (t >> 2) & 15, side = (group >> 1) & 1, c8 = (group >> 2) * 2 + (group & 1);
    reinterpret_cast<float4*>(xs)[(t & ~63) + (2 * v + side) * 8 + c8] = __ldg(reinterpret_cast<const float4*>(src) + t);
  }
}
// The sums of those sixteen elements, at block * 16 + side * 8 + c8: what the block minima multiply.
__device__ __forceinline__ void group_sums(const float* xs, float* sums, int count) {
  for (int t = threadIdx.x; t < count / 16; t += blockDim.x) {
    const float4* x = reinterpret_cast<const float4*>(xs) + (t >> 4) * 64 + (t & 15);
    float v = 0.0f;
#pragma unroll
    for (int i = 0; i < 4; ++i) v += (x[16 * i].x + x[16 * i].y) + (x[16 * i].z + x[16 * i].w);
    sums[t] = v;
  }
}

// What lane (c8 = lane % 8) contributes to the dot of one Q4_K block with 256 activations at
// `a` (staged by stage_activations; `sums`: group_sums of them): 16-byte chunk c8 of the nibble bytes (group g = c8/2: low nibbles -> elements
// 64g + 16(c8&1) + e, high nibbles -> +32, src/core/numerics/quant.cpp:656-675), from the
// block's header and that chunk, both already loaded.  A nibble becomes a float by the low mantissa bits of 2^23 (a byte
// permute and a subtraction): the conversion instruction runs at a sixteenth of the rate and bound the kernel.
__device__ __forceinline__ float q4k_chunk_dot(const float* a, const float* sums, uint4 hdr, uint4 q, int c8) {
  const int g = c8 >> 1;
  const float d = fp16_bits_to_float(hdr.x & 0xFFFFu);
  const float dmin = fp16_bits_to_float(hdr.x >> 16);
  // pairs 2g and 2g + 1 of the 12 packed bytes (q4k_scale_min) by shifts
  const int sh = 16 * (g & 1);
  const uint32_t s0 = hdr.y >> sh, s1 = hdr.z >> sh, s2 = hdr.w >> sh;
  const bool low = g < 2;
  const uint32_t sc0 = low ? s0 & 63u : (s2 & 15u) | ((s0 >> 2) & 48u), sc1 = low ? (s0 >> 8) & 63u : ((s2 >> 8) & 15u) | ((s0 >> 10) & 48u);
  const uint32_t mn0 = low ? s1 & 63u : ((s2 >> 4) & 15u) | ((s1 >> 2) & 48u), mn1 = low ? (s1 >> 8) & 63u : ((s2 >> 12) & 15u) | ((s1 >> 10) & 48u);
  const uint32_t qw[4] = {q.x, q.y, q.z, q.w};
  const float4* alo = reinterpret_cast<const float4*>(a) + c8;
  const float4* ahi = alo + 8;
  float sql = 0.f, sqh = 0.f;
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    const float4 x = alo[16 * v], y = ahi[16 * v];
    const float xs[4] = {x.x, x.y, x.z, x.w}, ys[4] = {y.x, y.y, y.z, y.w};
    const uint32_t lo = qw[v] & 0x0F0F0F0Fu, hi = (qw[v] >> 4) & 0x0F0F0F0Fu;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      sql = fmaf(__uint_as_float(__byte_perm(lo, 0x4B000000u, 0x7540 + e)) - 8388608.0f, xs[e], sql);
      sqh = fmaf(__uint_as_float(__byte_perm(hi, 0x4B000000u, 0x7540 + e)) - 8388608.0f, ys[e], sqh);
    }
  }
  const float sl = sums[c8], sum_h = sums[8 + c8];
  return d * static_cast<float>(sc0) * sql - dmin * static_cast<float>(mn0) * sl + d * static_cast<float>(sc1) * sqh -
         dmin * static_cast<float>(mn1) * sum_h;
}

// The same for one Q6_K block (210 bytes, 2-byte aligned): lane (h = lane/16, j = lane%16)
// takes elements 128h + 32r + 2j + {0,1}, r = 0..3 (src/core/numerics/quant.cpp:421-449).
__device__ __forceinline__ float q6k_block_share(const float* a, const uint8_t* block, int lane) {
  const int h = lane >> 4, j = lane & 15;
  constexpr float kMagic = 8388608.0f + 32.0f;  // (q | 0x4B000000) - kMagic = q - 32
  const unsigned short* blk = reinterpret_cast<const unsigned short*>(block);
  const uint32_t l0 = __ldg(blk + 32 * h + j), l1 = __ldg(blk + 32 * h + 16 + j), qh = __ldg(blk + 64 + 16 * h + j);
  const float d = fp16_bits_to_float(__ldg(blk + 104));
  const uint32_t s01 = __ldg(blk + 96 + 4 * h + 0), s23 = __ldg(blk + 96 + 4 * h + 1);
  const uint32_t s45 = __ldg(blk + 96 + 4 * h + 2), s67 = __ldg(blk + 96 + 4 * h + 3);
  const int sh = 8 * (j >> 3);
  const uint32_t sw[4] = {s01, s23, s45, s67};
  const float* ar = a + 128 * h + 2 * j;
  float acc = 0.0f;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const uint32_t lw = (r & 1) ? l1 : l0;
    const uint32_t nib = (r & 2) ? (lw >> 4) : lw;
    const uint32_t hi2 = qh >> (2 * r);
    const uint32_t q0 = (nib & 0xFu) | ((hi2 & 3u) << 4);
    const uint32_t q1 = ((nib >> 8) & 0xFu) | (((hi2 >> 8) & 3u) << 4);
    const float ds = d * static_cast<float>(static_cast<signed char>((sw[r] >> sh) & 0xFF));
    const float2 x = *reinterpret_cast<const float2*>(ar + 32 * r);
    acc = fmaf(x.x, ds * (__uint_as_float(q0 | 0x4B000000u) - kMagic), acc);
    acc = fmaf(x.y, ds * (__uint_as_float(q1 | 0x4B000000u) - kMagic), acc);
  }
  return acc;
}

// phi[slot][j] = silu(G_e[j] . x) * (U_e[j] . x), e = ids[slot]: one warp per (slot, j), x and its
// group sums in shared memory (dynamic: hidden + hidden / 16 floats).
__global__ void __launch_bounds__(kMoeWarps * 32)
moe_gate_up_q4k_kernel(const float* __restrict__ x, const uint8_t* __restrict__ gate, const uint8_t* __restrict__ up,
                       const uint32_t* __restrict__ ids, float* __restrict__ phi, int hidden, int inter, int top_k,
                       size_t gate_stride, size_t up_stride, int experts) {
  extern __shared__ __align__(16) float xs[];
  float* const sums = xs + hidden;
  const int idx = blockIdx.x * kMoeWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const bool have = idx < inter * top_k;
  const int slot = have ? idx / inter : 0, j = idx - slot * inter;
  const uint32_t e = have ? __ldg(ids + slot) : 0xFFFFFFFFu;
  const bool live = e < static_cast<uint32_t>(experts);  // an id outside the tensors: write nothing wrong, read nothing wild
  const int nb = live ? hidden / kBlockElems : 0;
  const size_t row = static_cast<size_t>(j) * (hidden / kBlockElems) * kQ4KBlockBytes;
  const uint8_t* grow = gate + (live ? e * gate_stride + row : 0);
  const uint8_t* urow = up + (live ? e * up_stride + row : 0);
  // lane (sub = lane/8, c8 = lane%8): chunk c8 of blocks sub, sub + 4, ...; the loads of two rounds of both rows are in
  // flight before the first is used, and those of the first two while x is being staged: they wait for the ids and then
  // for rows all over the expert tensors, which is most of the kernel's time
  const int sub = lane >> 3, c8 = lane & 7;
  uint4 hg[2], qg[2], hu[2], qu[2];
  auto fetch = [&](int b0) {
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int b = b0 + 4 * r;
      if (b < nb) {
        const uint8_t* gb = grow + static_cast<size_t>(b) * kQ4KBlockBytes;
        const uint8_t* ub = urow + static_cast<size_t>(b) * kQ4KBlockBytes;
        hg[r] = __ldg(reinterpret_cast<const uint4*>(gb));
        qg[r] = __ldg(reinterpret_cast<const uint4*>(gb + 16 + c8 * 16));
        hu[r] = __ldg(reinterpret_cast<const uint4*>(ub));
        qu[r] = __ldg(reinterpret_cast<const uint4*>(ub + 16 + c8 * 16));
      }
    }
  };
  fetch(sub);
  stage_activations(xs, x, hidden);
  __syncthreads();
  group_sums(xs, sums, hidden);
  __syncthreads();
  if (!have) return;
  float g = 0.0f, u = 0.0f;
  for (int b0 = sub; b0 < nb; b0 += 8) {
    if (b0 != sub) fetch(b0);
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int b = b0 + 4 * r;
      if (b < nb) {
        g += q4k_chunk_dot(xs + b * kBlockElems, sums + b * 16, hg[r], qg[r], c8);
        u += q4k_chunk_dot(xs + b * kBlockElems, sums + b * 16, hu[r], qu[r], c8);
      }
    }
  }
  g = warp_sum(g);
  u = warp_sum(u);
  if (lane == 0) phi[idx] = live ? (g / (1.0f + expf(-g))) * u : 0.0f;
}

// out[j] (+)= sum_slot wts[slot] * (D_e[j] . phi[slot]): one warp per j; phi (top_k x inter)
// and (Q4_K) its group sums in shared memory.
template <bool Q6>
__global__ void __launch_bounds__(kMoeWarps * 32)
moe_down_kernel(const float* __restrict__ phi, const uint8_t* __restrict__ down, const uint32_t* __restrict__ ids,
                const float* __restrict__ wts, float* __restrict__ out, int hidden, int inter, int top_k,
                size_t down_stride, int accumulate, int experts) {
  extern __shared__ __align__(16) float ps[];
  float* const sums = ps + top_k * inter;
  const int j = blockIdx.x * kMoeWarps + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int nb = inter / kBlockElems;
  // Q4_K: the (slot, block) pairs of this output row, four at a time across the warp (lane/8) and
  // two such rounds in flight: the row of an expert is short (inter/256 blocks); the first rounds are asked for before
  // the staging
  const int sub = lane >> 3, c8 = lane & 7, pairs = j < hidden ? top_k * nb : 0;
  constexpr int kRounds = Q6 ? 1 : 4;
  uint4 h[kRounds], q[kRounds];
  float w[kRounds];
  int at[kRounds];
  auto fetch = [&](int p0) {
#pragma unroll
    for (int r = 0; r < kRounds; ++r) {
      const int pr = p0 + 4 * r;
      w[r] = 0.0f;
      at[r] = 0;
      h[r] = q[r] = make_uint4(0u, 0u, 0u, 0u);
      if (pr < pairs) {
        const int slot = pr / nb, b = pr - slot * nb;
        const uint32_t e = __ldg(ids + slot);
        if (e < static_cast<uint32_t>(experts)) {
          const uint8_t* blk = down + e * down_stride + (static_cast<size_t>(j) * nb + b) * kQ4KBlockBytes;
          h[r] = __ldg(reinterpret_cast<const uint4*>(blk));
          q[r] = __ldg(reinterpret_cast<const uint4*>(blk + 16 + c8 * 16));
          w[r] = __ldg(wts + slot);
          at[r] = slot * inter + b * kBlockElems;
        }
      }
    }
  };
  if (!Q6) fetch(sub);
  if (Q6) {
    for (int t = threadIdx.x; t < top_k * inter / 4; t += blockDim.x)
      reinterpret_cast<float4*>(ps)[t] = __ldg(reinterpret_cast<const float4*>(phi) + t);
  } else {
    stage_activations(ps, phi, top_k * inter);
  }
  __syncthreads();
  if (!Q6) {
    group_sums(ps, sums, top_k * inter);
    __syncthreads();
  }
  if (j >= hidden) return;
  float acc = 0.0f;
  if (Q6) {
    // a whole warp per block; two (slot, block) pairs are loaded before the first is used
    for (int slot = 0; slot < top_k; ++slot) {
      const uint32_t e = ids[slot];
      if (e >= static_cast<uint32_t>(experts)) continue;
      const uint8_t* row = down + e * down_stride + static_cast<size_t>(j) * nb * kQ6KBlockBytes;
      float part = 0.0f;
#pragma unroll 2
      for (int b = 0; b < nb; ++b)
        part += q6k_block_share(ps + slot * inter + b * kBlockElems, row + static_cast<size_t>(b) * kQ6KBlockBytes, lane);
      acc = fmaf(wts[slot], part, acc);
    }
  } else {
    for (int p0 = sub; p0 < pairs; p0 += 4 * kRounds) {
      if (p0 != sub) fetch(p0);
#pragma unroll
      for (int r = 0; r < kRounds; ++r) acc = fmaf(w[r], q4k_chunk_dot(ps + at[r], sums + at[r] / 16, h[r], q[r], c8), acc);
    }
  }
  acc = warp_sum(acc);
  if (lane == 0) out[j] = accumulate ? out[j] + acc : acc;
}

__global__ void __launch_bounds__(kRouterThreads)
moe_gate_kernel(const float* __restrict__ vals, const float* __restrict__ x, const float* __restrict__ w,
                float* __restrict__ wts, float* __restrict__ sig, int top_k, int hidden) {
  __shared__ float red[kRouterThreads / 32];
  moe_gate_dot(x, w, hidden, red);
  __syncthreads();
  moe_gate_finish(vals, wts, sig, top_k, red);
}

// top_k_rows and moe_gate of one token in one launch (the queue finds them side by side): same arithmetic and order.
template <int P>
__global__ void __launch_bounds__(kRouterThreads)
router_select_kernel(const float* __restrict__ logits, uint32_t* ids, float* vals,
                     const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ wts,
                     float* __restrict__ sig, int vocab, int top_k, int hidden) {
  __shared__ TopKShared shared;
  __shared__ float red[kRouterThreads / 32];
  top_k_small<P>(logits, ids, vals, vocab, top_k, shared, [&] { moe_gate_dot(x, w, hidden, red); });
  __syncthreads();
  moe_gate_finish(shared.chosen, wts, sig, top_k, red);
}

__global__ void moe_scale_add_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                     const float* __restrict__ f, float* __restrict__ o, size_t n, size_t idx) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) o[i] = __fadd_rn(a[i], __fmul_rn(f[idx], b[i]));  // two roundings, as the contract's expression reads
}

// The same followed by `add` with its result (out = base + (a + f[idx] b)), both results written.
__global__ void moe_scale_add_add_kernel(const float* __restrict__ a, const float* __restrict__ b, const float* __restrict__ f,
                                         float* __restrict__ o, const float* base, float* out, size_t n, size_t idx) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float v = __fadd_rn(a[i], __fmul_rn(f[idx], b[i]));
  o[i] = v;
  out[i] = __fadd_rn(base[i], v);
}

bool fits31(uint64_t v) { return v > 0 && v <= 0x7FFFFFFFull; }
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

int launch_router_select(const float* logits, uint32_t* ids, float* vals, const float* x, const float* w, float* wts, float* sig,
                         uint64_t vocab, uint64_t top_k, uint64_t hidden, cudaStream_t st) {
  if (vocab > kTopKSmall || top_k == 0 || top_k > 32 || !fits31(vocab) || !fits31(hidden)) return kUnsupportedFeature;
  const int v = static_cast<int>(vocab), t = static_cast<int>(top_k), h = static_cast<int>(hidden);
  if (vocab <= 128) router_select_kernel<4><<<1, kRouterThreads, 0, st>>>(logits, ids, vals, x, w, wts, sig, v, t, h);
  else if (vocab <= 256) router_select_kernel<8><<<1, kRouterThreads, 0, st>>>(logits, ids, vals, x, w, wts, sig, v, t, h);
  else router_select_kernel<32><<<1, kRouterThreads, 0, st>>>(logits, ids, vals, x, w, wts, sig, v, t, h);
  return check_launch();
}
int launch_moe_scale_add_add(const float* a, const float* b, const float* f, float* o, const float* base, float* out, uint64_t n,
                             uint64_t idx, cudaStream_t st) {
  moe_scale_add_add_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(a, b, f, o, base, out, n, idx);
  return check_launch();
}

}  // namespace tsr

using namespace tsr;

extern "C" {

int tsr_moe_gate(const float* vals, const float* x, const float* w, float* wts, float* sig, uint64_t top_k,
                 uint64_t hidden, void* stream) {
  if (!vals || !x || !w || !wts || !sig || !fits31(top_k) || !fits31(hidden)) return kInvalidArgument;
  moe_gate_kernel<<<1, kRouterThreads, 0, static_cast<cudaStream_t>(stream)>>>(vals, x, w, wts, sig, static_cast<int>(top_k),
                                                                     static_cast<int>(hidden));
  return check_launch();
}

int tsr_moe_scale_add(const float* a, const float* b, const float* f, float* o, uint64_t n, uint64_t idx, void* stream) {
  if (!a || !b || !f || !o || n == 0) return kInvalidArgument;
  moe_scale_add_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(a, b, f, o, n,
                                                                                                                   idx);
  return check_launch();
}

int tsr_moe_experts_gate_up_q4k(const float* x, const void* gate, const void* up, const uint32_t* ids, float* phi,
                                uint64_t hidden, uint64_t inter, uint64_t top_k, uint64_t gate_stride, uint64_t up_stride,
                                uint64_t experts, void* stream) {
  if (!x || !gate || !up || !ids || !phi || !fits31(hidden) || !fits31(inter) || !fits31(top_k) || !fits31(experts) ||
      hidden % 256 != 0 || !fits31(inter * top_k) || hidden * 4 > 200 * 1024)
    return kInvalidArgument;
  if (!aligned16(x) || !aligned16(gate) || !aligned16(up) || gate_stride % 16 != 0 || up_stride % 16 != 0)
    return kInvalidArgument;
  const size_t smem = hidden * 4 + hidden / 4;
  if (int rc = allow_dynamic_smem(reinterpret_cast<const void*>(&moe_gate_up_q4k_kernel), 227 * 1024)) return rc;
  const unsigned blocks = static_cast<unsigned>((inter * top_k + kMoeWarps - 1) / kMoeWarps);
  moe_gate_up_q4k_kernel<<<blocks, kMoeWarps * 32, smem, static_cast<cudaStream_t>(stream)>>>(
      x, static_cast<const uint8_t*>(gate), static_cast<const uint8_t*>(up), ids, phi, static_cast<int>(hidden),
      static_cast<int>(inter), static_cast<int>(top_k), gate_stride, up_stride, static_cast<int>(experts));
  return check_launch();
}

int tsr_moe_experts_down(int fmt, const float* phi, const void* down, const uint32_t* ids, const float* wts, float* out,
                         uint64_t hidden, uint64_t inter, uint64_t top_k, uint64_t down_stride, uint64_t accumulate,
                         uint64_t experts, void* stream) {
  if ((fmt != 0 && fmt != 1) || !phi || !down || !ids || !wts || !out || !fits31(hidden) || !fits31(inter) ||
      !fits31(top_k) || !fits31(experts) || inter % 256 != 0 || top_k * inter * 4 > 200 * 1024)
    return kInvalidArgument;
  if (!aligned16(phi) || (fmt == 0 && (!aligned16(down) || down_stride % 16 != 0)) ||
      (fmt == 1 && ((reinterpret_cast<uintptr_t>(down) & 1u) || down_stride % 2 != 0)))
    return kInvalidArgument;
  const size_t smem = top_k * inter * 4 + top_k * inter / 4;
  const unsigned blocks = static_cast<unsigned>((hidden + kMoeWarps - 1) / kMoeWarps);
  auto st = static_cast<cudaStream_t>(stream);
  if (fmt == 0) {
    if (int rc = allow_dynamic_smem(reinterpret_cast<const void*>(&moe_down_kernel<false>), 227 * 1024)) return rc;
    moe_down_kernel<false><<<blocks, kMoeWarps * 32, smem, st>>>(phi, static_cast<const uint8_t*>(down), ids, wts, out,
                                                                  static_cast<int>(hidden), static_cast<int>(inter),
                                                                  static_cast<int>(top_k), down_stride,
                                                                  accumulate != 0 ? 1 : 0, static_cast<int>(experts));
  } else {
    if (int rc = allow_dynamic_smem(reinterpret_cast<const void*>(&moe_down_kernel<true>), 227 * 1024)) return rc;
    moe_down_kernel<true><<<blocks, kMoeWarps * 32, smem, st>>>(phi, static_cast<const uint8_t*>(down), ids, wts, out,
                                                                 static_cast<int>(hidden), static_cast<int>(inter),
                                                                 static_cast<int>(top_k), down_stride,
                                                                 accumulate != 0 ? 1 : 0, static_cast<int>(experts));
  }
  return check_launch();
}

}  // extern "C"
