// Small kernels around the projections: per-token FP8 activation
// quantisation, split-K reduce, bf16 rounding, add, fill, the MXFP4 row
// reference byte, and the bit-exact block dequantiser used by the codec
// parity tests.
#include "codec.cuh"
#include "launch.h"
#include "tessera_b200.h"

namespace tsr {

// ------------------------------------------------ per-token FP8 quantise
// One CTA per row.  scale = max(amax/448, 1/(448*512)); q = clamp(x/scale,
// +-448) coded to E4M3 round-to-nearest-even
// (src/core/numerics/quant.cpp:180-229).  PACK writes codes, else the data is
// replaced by code*scale in place.
template <bool PACK>
__global__ void __launch_bounds__(1024)
quantize_fp8_kernel(float* __restrict__ data, const float* __restrict__ in,
                    uint8_t* __restrict__ codes, float* __restrict__ scale, int cols) {
  __shared__ float red[32];
  const size_t base = static_cast<size_t>(blockIdx.x) * cols;
  const float* src = PACK ? in + base : data + base;
  float amax = 0.0f;
  for (int cidx = threadIdx.x; cidx < cols; cidx += blockDim.x)
    amax = fmaxf(amax, fabsf(src[cidx]));  // fmaxf drops NaN like std::max(amax, x)
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xFFFFFFFFu, v, o));
    if (threadIdx.x == 0) red[0] = v;
  }
  __syncthreads();
  const float s = fmaxf(__fdiv_rn(red[0], 448.0f), 1.0f / (448.0f * 512.0f));
  if (threadIdx.x == 0) scale[blockIdx.x] = s;
  for (int cidx = threadIdx.x; cidx < cols; cidx += blockDim.x) {
    float q = __fdiv_rn(src[cidx], s);
    q = q < -448.0f ? -448.0f : (448.0f < q ? 448.0f : q);  // std::clamp; NaN passes through
    const uint32_t code = float_to_e4m3_ref(q);
    if (PACK) {
      codes[base + cidx] = static_cast<uint8_t>(code);
    } else {
      data[base + cidx] = __fmul_rn(e4m3_to_float(code), s);
    }
  }
}

// The code float_to_e4m3_ref gives a value in [-448, 448] (or a NaN), from the hardware's conversion: both round to
// nearest even, but the reference clamps a subnormal's mantissa at 7 where rounding would carry into the smallest normal
// value, and keeps a NaN's sign.
__device__ __forceinline__ uint32_t e4m3_code(float q) {
  const uint32_t bits = __float_as_uint(q), sign = (bits >> 31) << 7;
  const float mag = fabsf(q);
  uint32_t code = __nv_cvt_float_to_fp8(q, __NV_SATFINITE, __NV_E4M3);
  if (mag >= 7.5f / 512.0f && mag < 8.0f / 512.0f) code = sign | 7u;
  return q == q ? code : (sign | 0x7Fu);
}

// The codes of a batch (quantize_fp8_pack) with several CTAs per row: each finds the row's maximum by itself (the row is
// a few tens of KB, served from L2 after the first) and codes its share, four columns a thread.  One CTA a row left 16
// verify rows on 16 SMs, with frexp and a 64-bit rounding an element: 16 rows of 5120 / 17408 took 7.3 / 17.6 us, here
// 4.3 / 4.7.
constexpr int kPackThreads = 512;
__global__ void __launch_bounds__(kPackThreads)
quantize_fp8_pack_kernel(const float4* __restrict__ in, uint32_t* __restrict__ codes, float* __restrict__ scale, int cols4) {
  __shared__ float red[kPackThreads / 32];
  const size_t base = static_cast<size_t>(blockIdx.x) * cols4;
  float amax = 0.0f;
#pragma unroll 4
  for (int c = threadIdx.x; c < cols4; c += kPackThreads) {
    const float4 x = __ldg(in + base + c);
    amax = fmaxf(amax, fmaxf(fmaxf(fabsf(x.x), fabsf(x.y)), fmaxf(fabsf(x.z), fabsf(x.w))));  // fmaxf drops NaN like std::max
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xFFFFFFFFu, amax, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = amax;
  __syncthreads();
  amax = red[0];
#pragma unroll
  for (int w = 1; w < kPackThreads / 32; ++w) amax = fmaxf(amax, red[w]);
  const float s = fmaxf(__fdiv_rn(amax, 448.0f), 1.0f / (448.0f * 512.0f));
  if (blockIdx.y == 0 && threadIdx.x == 0) scale[blockIdx.x] = s;
  const int share = (cols4 + gridDim.y - 1) / gridDim.y, c0 = blockIdx.y * share, c1 = min(cols4, c0 + share);
  for (int c = c0 + threadIdx.x; c < c1; c += kPackThreads) {
    const float4 x = __ldg(in + base + c);
    const float v[4] = {x.x, x.y, x.z, x.w};
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float q = __fdiv_rn(v[i], s);
      q = q < -448.0f ? -448.0f : (448.0f < q ? 448.0f : q);  // std::clamp; NaN passes through
      w |= e4m3_code(q) << (8 * i);
    }
    codes[base + c] = w;
  }
}

// gemm_vec_reduce.comp:20-32: ordered sum of the split regions.
__global__ void vec_reduce_kernel(const float* __restrict__ part, float* __restrict__ c,
                                  size_t total, int split) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  pdl_wait();     // the partials come from the kernel just ahead
  pdl_trigger();  // the next projection may start prefetching its weights
  if (i >= total) return;
  float acc = 0.0f;
  for (int s = 0; s < split; ++s) acc += part[s * total + i];
  c[i] = acc;
}

// round_bf16.comp:14-24 / quant.cpp:231-243.
__global__ void round_bf16_kernel(float* __restrict__ x, size_t n) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t u = __float_as_uint(x[i]);
  u += 0x7FFFu + ((u >> 16) & 1u);
  x[i] = __uint_as_float(u & 0xFFFF0000u);
}

__global__ void bf16_to_f32_kernel(const unsigned short* __restrict__ src, float* __restrict__ dst, size_t n) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) dst[i] = __uint_as_float(static_cast<uint32_t>(src[i]) << 16);
}

// the rounding of round_bf16_kernel, stored as the high half
__global__ void f32_to_bf16_kernel(const float* __restrict__ src, unsigned short* __restrict__ dst, size_t n) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n) return;
  uint32_t u = __float_as_uint(src[i]);
  u += 0x7FFFu + ((u >> 16) & 1u);
  dst[i] = static_cast<unsigned short>(u >> 16);
}

__global__ void add_kernel(const float* __restrict__ a, const float* __restrict__ b,
                           float* __restrict__ o, size_t n) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) o[i] = a[i] + b[i];
}

__global__ void fill_kernel(int32_t* __restrict__ d, int32_t v, size_t n) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i < n) d[i] = v;
}

// mxfp4_row_ref.comp:26-40: largest E8M0 byte of each row; warp per row.
__global__ void mxfp4_row_ref_kernel(const uint8_t* __restrict__ w, uint8_t* __restrict__ wref,
                                     int n, int k) {
  const int row = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (row >= n) return;
  const int nb = k / 32;
  const uint8_t* s = w + static_cast<size_t>(n) * (k / 2) + static_cast<size_t>(row) * nb;
  uint32_t mx = 0;
  for (int b = threadIdx.x & 31; b < nb; b += 32) mx = max(mx, static_cast<uint32_t>(s[b]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = max(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
  if ((threadIdx.x & 31) == 0) wref[row] = static_cast<uint8_t>(mx);
}

// Bit-exact dequantiser: one thread per element, every product and the
// subtraction rounded separately, as the host reference does without fused
// multiply-add.
__global__ void dequantize_kernel(int fmt, const uint8_t* __restrict__ w,
                                  const float* __restrict__ row_scale, float* __restrict__ out,
                                  size_t n, size_t k) {
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= n * k) return;
  const size_t row = idx / k, t = idx % k;
  float v = 0.0f;
  if (fmt == 0) {
    const uint8_t* blk = w + (row * (k / 256) + t / 256) * kQ4KBlockBytes;
    const int e = static_cast<int>(t % 256), g = e / 64, hi = (e % 64) / 32, l = e % 32;
    const float d = fp16_bits_to_float(blk[0] | (blk[1] << 8));
    const float dmin = fp16_bits_to_float(blk[2] | (blk[3] << 8));
    uint32_t s[3];
    for (int i = 0; i < 3; ++i)
      s[i] = blk[4 + 4 * i] | (blk[5 + 4 * i] << 8) | (blk[6 + 4 * i] << 16) |
             (static_cast<uint32_t>(blk[7 + 4 * i]) << 24);
    uint32_t sc, mn;
    q4k_scale_min(s, 2 * g + hi, sc, mn);
    const uint32_t byte = blk[16 + 32 * g + l];
    const float q = static_cast<float>(hi ? (byte >> 4) : (byte & 15u));
    v = __fsub_rn(__fmul_rn(__fmul_rn(d, static_cast<float>(sc)), q),
                  __fmul_rn(dmin, static_cast<float>(mn)));
  } else if (fmt == 1) {
    const uint8_t* blk = w + (row * (k / 256) + t / 256) * kQ6KBlockBytes;
    const int e = static_cast<int>(t % 256), h = e / 128, part = (e % 128) / 32, l = e % 32;
    const float d = fp16_bits_to_float(blk[208] | (blk[209] << 8));
    const uint32_t lo = blk[64 * h + 32 * (part & 1) + l];
    const uint32_t qh = blk[128 + 32 * h + l];
    const uint32_t nib = (part & 2) ? (lo >> 4) : (lo & 15u);
    const int q = static_cast<int>(nib | (((qh >> (2 * part)) & 3u) << 4)) - 32;
    const float sc = static_cast<float>(static_cast<signed char>(blk[192 + 8 * h + l / 16 + 2 * part]));
    v = __fmul_rn(__fmul_rn(d, sc), static_cast<float>(q));
  } else if (fmt == 2) {
    const uint32_t byte = w[(row * k + t) / 2];
    const uint32_t nib = (t % 2 == 0) ? (byte & 15u) : (byte >> 4);
    const uint32_t sb = w[n * (k / 2) + row * (k / 32) + t / 32];
    v = __fmul_rn(e8m0_to_float(sb), e2m1_to_float(nib));
  } else {
    v = __fmul_rn(row_scale[row], e4m3_to_float(w[row * k + t]));
  }
  out[idx] = v;
}

// O = silu(G) * U (SiluMulRef, src/core/numerics/norm.cpp:211-225)
__global__ void silu_mul_kernel(const float* __restrict__ g, const float* __restrict__ u, float* __restrict__ o,
                                size_t n) {
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= n) return;
  const float x = g[idx];
  o[idx] = x / (1.0f + expf(-x)) * u[idx];
}

// The same and `add`, sixteen bytes a load (n a multiple of four, 16-byte aligned buffers): an element a thread kept too
// few bytes in flight for a prompt chunk (512 x 17408, operands from memory: silu_mul 40 us, here 18.7 us = 5.7 TB/s; 15 us
// where the two projections have left part of them in L2).
__global__ void __launch_bounds__(256) silu_mul4_kernel(const float4* g, const float4* u,
                                                        float4* o, size_t n4) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const float4 x = g[i], y = u[i];
  o[i] = make_float4(x.x / (1.0f + expf(-x.x)) * y.x, x.y / (1.0f + expf(-x.y)) * y.y, x.z / (1.0f + expf(-x.z)) * y.z,
                     x.w / (1.0f + expf(-x.w)) * y.w);
}
__global__ void __launch_bounds__(256) add4_kernel(const float4* a, const float4* b, float4* o, size_t n4) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= n4) return;
  const float4 x = a[i], y = b[i];
  o[i] = make_float4(x.x + y.x, x.y + y.y, x.z + y.z, x.w + y.w);
}

// Y = X / sqrt(mean(X^2) + eps) * W, one CTA per row (RmsNormRef, src/core/numerics/norm.cpp:7-32;
// the reference adds the squares sequentially, here they are added as a tree).
__global__ void __launch_bounds__(1024)
rmsnorm_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int cols, float eps) {
  __shared__ float red[32];
  constexpr int kHeld = 8;  // of a thread's columns, the first eight stay in registers: their loads are in flight together
  const float* row = x + static_cast<size_t>(blockIdx.x) * cols;
  float held[kHeld], weight[kHeld];
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    held[i] = c < cols ? row[c] : 0.0f;
    weight[i] = c < cols ? __ldg(w + c) : 0.0f;
  }
  float s = 0.0f;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) s = fmaf(held[i], held[i], s);
  for (int c = threadIdx.x + kHeld * blockDim.x; c < cols; c += blockDim.x) s = fmaf(row[c], row[c], s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    float v = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    if (threadIdx.x == 0) red[0] = 1.0f / sqrtf(v / static_cast<float>(cols) + eps);
  }
  __syncthreads();
  const float gain = red[0];
  float* out = y + static_cast<size_t>(blockIdx.x) * cols;
#pragma unroll
  for (int i = 0; i < kHeld; ++i) {
    const int c = threadIdx.x + i * blockDim.x;
    if (c < cols) out[c] = held[i] * gain * weight[i];
  }
  for (int c = threadIdx.x + kHeld * blockDim.x; c < cols; c += blockDim.x) out[c] = row[c] * gain * w[c];
}

// Whether an elementwise step over n floats takes the four-wide kernel: from 256k elements on (below, a quarter of the
// threads is a quarter of the SMs), whole and aligned, and with an output that is one of the inputs or apart from them (a
// thread reads four elements before it writes four).
static bool wide4(const float* a, const float* b, const float* o, uint64_t n) {
  auto apart = [&](const float* x) { return x == o || o + n <= x || x + n <= o; };
  return n >= (1u << 18) && n % 4 == 0 && ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(o)) & 15u) == 0 &&
         apart(a) && apart(b);
}
static unsigned blocks_for(uint64_t n, unsigned per) {
  return static_cast<unsigned>((n + per - 1) / per);
}

int convert_bf16_to_f32(const void* src, float* dst, uint64_t n, cudaStream_t st) {
  bf16_to_f32_kernel<<<blocks_for(n, 256), 256, 0, st>>>(static_cast<const unsigned short*>(src), dst, n);
  return check_launch();
}
int convert_f32_to_bf16(const float* src, void* dst, uint64_t n, cudaStream_t st) {
  f32_to_bf16_kernel<<<blocks_for(n, 256), 256, 0, st>>>(src, static_cast<unsigned short*>(dst), n);
  return check_launch();
}

}  // namespace tsr

using namespace tsr;

extern "C" {

int tsr_quantize_fp8(float* data, float* scale, uint64_t rows, uint64_t cols, void* stream) {
  if (!data || !scale || rows == 0 || cols == 0 || cols > 0x7FFFFFFFull) return kInvalidArgument;
  quantize_fp8_kernel<false><<<static_cast<unsigned>(rows), 1024, 0,
                               static_cast<cudaStream_t>(stream)>>>(data, nullptr, nullptr, scale,
                                                                    static_cast<int>(cols));
  return check_launch();
}

int tsr_quantize_fp8_pack(const float* in, void* out, float* scale, uint64_t rows, uint64_t cols,
                          void* stream) {
  if (!in || !out || !scale || rows == 0 || cols == 0 || cols % 4 != 0 || cols > 0x7FFFFFFFull)
    return kInvalidArgument;
  if (((reinterpret_cast<uintptr_t>(in) & 15u) | (reinterpret_cast<uintptr_t>(out) & 3u)) == 0 && rows <= 0x7FFFFFFFull) {
    // CTAs per row: up to two per SM over all rows, at least 1024 columns each
    const uint64_t most = (cols + 1023) / 1024, want = (296 + rows - 1) / rows;
    const unsigned parts = static_cast<unsigned>(want < most ? want : most);
    quantize_fp8_pack_kernel<<<dim3(static_cast<unsigned>(rows), parts), kPackThreads, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const float4*>(in), static_cast<uint32_t*>(out), scale, static_cast<int>(cols / 4));
    return check_launch();
  }
  quantize_fp8_kernel<true><<<static_cast<unsigned>(rows), 1024, 0,
                              static_cast<cudaStream_t>(stream)>>>(
      nullptr, in, static_cast<uint8_t*>(out), scale, static_cast<int>(cols));
  return check_launch();
}

int tsr_gemm_vec_reduce(const float* part, float* c, uint64_t total, uint64_t split, void* stream) {
  if (!part || !c || total == 0 || split == 0) return kInvalidArgument;
  auto st = static_cast<cudaStream_t>(stream);
  // reads the partial buffer only after its wait, so it can always be a programmatic dependent
  const bool pdl = pdl_allowed(st, nullptr, 0, c, total * 4);
  launch_kernel(vec_reduce_kernel, dim3(blocks_for(total, 256)), dim3(256), 0, st, pdl, part, c,
                static_cast<size_t>(total), static_cast<int>(split));
  return check_launch();
}

int tsr_round_bf16(float* x, uint64_t n, void* stream) {
  if (!x || n == 0) return kInvalidArgument;
  round_bf16_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, n);
  return check_launch();
}

int tsr_add(const float* a, const float* b, float* o, uint64_t n, void* stream) {
  if (!a || !b || !o || n == 0) return kInvalidArgument;
  if (wide4(a, b, o, n)) {
    add4_kernel<<<blocks_for(n / 4, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        reinterpret_cast<const float4*>(a), reinterpret_cast<const float4*>(b), reinterpret_cast<float4*>(o), n / 4);
    return check_launch();
  }
  add_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(a, b, o, n);
  return check_launch();
}

int tsr_silu_mul(const float* g, const float* u, float* o, uint64_t n, void* stream) {
  if (!g || !u || !o || n == 0) return kInvalidArgument;
  auto st = static_cast<cudaStream_t>(stream);
  if (wide4(g, u, o, n))
    silu_mul4_kernel<<<blocks_for(n / 4, 256), 256, 0, st>>>(reinterpret_cast<const float4*>(g), reinterpret_cast<const float4*>(u),
                                                             reinterpret_cast<float4*>(o), n / 4);
  else
    silu_mul_kernel<<<blocks_for(n, 256), 256, 0, st>>>(g, u, o, n);
  return check_launch();
}

int tsr_rmsnorm(const float* x, const float* w, float* y, uint64_t rows, uint64_t cols, float eps, void* stream) {
  if (!x || !w || !y || rows == 0 || cols == 0 || rows > 0x7FFFFFFFull || cols > 0x7FFFFFFFull || !(eps >= 0.0f))
    return kInvalidArgument;
  rmsnorm_kernel<<<static_cast<unsigned>(rows), cols >= 4096 ? 1024 : 256, 0, static_cast<cudaStream_t>(stream)>>>(
      x, w, y, static_cast<int>(cols), eps);
  return check_launch();
}

int tsr_fill(int32_t* data, int32_t value, uint64_t n, void* stream) {
  if (!data || n == 0) return kInvalidArgument;
  fill_kernel<<<blocks_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(data, value, n);
  return check_launch();
}

int tsr_mxfp4_row_ref(const void* w, void* wref, uint64_t n, uint64_t k, void* stream) {
  if (!w || !wref || n == 0 || k == 0 || k % 32 != 0) return kInvalidArgument;
  mxfp4_row_ref_kernel<<<blocks_for(n, 8), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      static_cast<const uint8_t*>(w), static_cast<uint8_t*>(wref), static_cast<int>(n),
      static_cast<int>(k));
  return check_launch();
}

int tsr_dequantize(int fmt, const void* w, const float* row_scale, float* out, uint64_t n,
                   uint64_t k, void* stream) {
  if (!w || !out || n == 0 || k == 0 || fmt < 0 || fmt > 3) return kInvalidArgument;
  if ((fmt <= 1 && k % 256 != 0) || (fmt == 2 && k % 32 != 0) || (fmt == 3 && !row_scale))
    return kInvalidArgument;
  dequantize_kernel<<<blocks_for(n * k, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
      fmt, static_cast<const uint8_t*>(w), row_scale, out, n, k);
  return check_launch();
}

}  // extern "C"
