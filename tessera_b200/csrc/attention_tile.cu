// Grouped-query attention of a batch of query rows (prompt chunks, speculative-verify batches) over a 16-bit or
// narrower key / value cache, on the tensor pipe.  Contract, masks and arithmetic are those of attention.cu (ids
// "attention" with an fp16 cache, "attention_q8" / "_q4" / "_fp8"; AttentionRefF16, AttentionQ8Ref, AttentionQ4Ref,
// AttentionFp8Ref, src/core/numerics/attention.cpp of the reference).
//
// The chunk kernel of attention.cu serves one query row per CTA: a batch of 512 rows re-read the cache 512 times,
// ran 2 x 24 GFLOP (4096 keys, 24 heads of 256) as fp32 multiply-adds and wrote 805 MB of partial sums.  Here a CTA
// takes 128 (query row, head) pairs of one kv head and walks over tiles of 64 keys.  Both products are contractions,
// so they run as m16n8k16 binary16 MMAs with fp32 accumulation.  Nothing is rounded to 16 bits on the way: cache
// elements (FP8, int8, 4-bit, fp16) are exact in binary16, and a query element or a softmax weight enters as two
// binary16 terms x = hi + lo of a value scaled by a power of two, 22 bits below the row's largest query element and
// 2^-38 below the row's largest weight.  Scales of quantised rows multiply the score and the weight in fp32.  The MMA
// cuts off what falls below its accumulator instead of rounding (chains over 4096 keys came out 4e-6 off), so two MMAs
// of a score and eight of an output share an accumulator, the small terms first, before it is added in fp32: 3.8e-7
// against 64 bits where the chunk kernel's fp32 sums have 3.0e-7 (longer chains 4.9e-7 at 6 % less time).
//
// mma.sync rather than tcgen05: the 128 x 256 output accumulators have to be rescaled whenever a row's maximum
// grows, which registers do in place and tensor memory only by a round trip; the two-term queries (128 KB) leave no
// shared memory for the weights as a tcgen05 operand.
// Bound: the tensor pipe, at the mma.sync rate: four MMAs where a plain product needs two.  512 rows over 4096 FP8 keys,
// 24 heads of 256: 394 us against 4470 (123 TFLOP/s of the contract's 48 GFLOP, 246 of the MMAs').
#include <cuda_fp16.h>

#include "attention.cuh"
#include "codec.cuh"
#include "launch.h"

namespace tsr {
namespace {

constexpr int kTileRows = 128, kTileKeys = 64, kTileThreads = 256;
constexpr int kScoreChain = 1, kValueChain = 4;  // 16-wide k steps (of two MMAs) that share an accumulator
constexpr int kWeightBits = 14;  // softmax weights (<= 1) and normalised value scales are stored times 2^14

struct AttnTileParams {
  AttnParams a;
  float* out;         // with one split: the result itself
  const float* gate;  // out *= sigmoid(gate), or null
  int group, row_tiles, tiles_per_split;
};

template <int KV, int D>
struct TileShape {
  static constexpr int kRowBytes = D * kv_bits<KV>() / 8;                 // a cache row of one kv head
  static constexpr int kPiecesPerRow = kRowBytes / 16;
  static constexpr int kPieces = kTileKeys * kPiecesPerRow / kTileThreads;  // 16-byte pieces a thread moves per tile
  static constexpr int kQBytes = 2 * kTileRows * D * 2, kTileBytes = kTileKeys * D * 2;
  static constexpr int kRawBytes = KV == kKvF16 ? 0 : kTileKeys * kRowBytes;
  static constexpr int kSmem = kQBytes + 2 * kTileBytes + 2 * kRawBytes + kTileRows * 4 + 2 * 2 * kTileKeys * 4 + 64;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldmatrix4_trans(uint32_t (&r)[4], uint32_t addr) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void mma_f16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_half2(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
// (x, y) as binary16 and what binary16 lost of them
__device__ __forceinline__ void split_half2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  hi = pack_half2(h);
  lo = pack_half2(__floats2half2_rn(x - f.x, y - f.y));
}
__device__ __forceinline__ __half2 u32_half2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }

// A 16-byte piece of the cache as binary16 values; true when an element is not finite.
__device__ __forceinline__ bool has_nonfinite_fp8(uint32_t w) { return (((w & 0x7F7F7F7Fu) + 0x01010101u) & 0x80808080u) != 0; }
__device__ __forceinline__ bool has_nonfinite_f16(uint32_t w) { return (((w & 0x7C007C00u) + 0x04000400u) & 0x80008000u) != 0; }

template <int KV>
__device__ __forceinline__ bool expand_word(uint32_t w, uint32_t (&h)[KV == kKvInt4 ? 4 : 2]) {
  if constexpr (KV == kKvFp8) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const __half2_raw r = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>((w >> (16 * i)) & 0xFFFFu), __NV_E4M3);
      h[i] = pack_half2(__half2(r));
    }
    return has_nonfinite_fp8(w);
  } else if constexpr (KV == kKvInt8) {  // 1024 + (b + 128) - 1152, exact
    const uint32_t u = w ^ 0x80808080u;
    h[0] = pack_half2(__hsub2(u32_half2(__byte_perm(u, 0x64646464u, 0x4140)), u32_half2(0x64806480u)));
    h[1] = pack_half2(__hsub2(u32_half2(__byte_perm(u, 0x64646464u, 0x4342)), u32_half2(0x64806480u)));
    return false;
  } else {  // two's-complement nibbles, element 2i low: 1024 + (v + 8) - 1032
    const uint32_t t = w ^ 0x88888888u, even = t & 0x0F0F0F0Fu, odd = (t >> 4) & 0x0F0F0F0Fu;
    const uint32_t x = __byte_perm(even, odd, 0x5140), y = __byte_perm(even, odd, 0x7362);
    h[0] = pack_half2(__hsub2(u32_half2(__byte_perm(x, 0x64646464u, 0x4140)), u32_half2(0x64086408u)));
    h[1] = pack_half2(__hsub2(u32_half2(__byte_perm(x, 0x64646464u, 0x4342)), u32_half2(0x64086408u)));
    h[2] = pack_half2(__hsub2(u32_half2(__byte_perm(y, 0x64646464u, 0x4140)), u32_half2(0x64086408u)));
    h[3] = pack_half2(__hsub2(u32_half2(__byte_perm(y, 0x64646464u, 0x4342)), u32_half2(0x64086408u)));
    return false;
  }
}

// Cache element e of a row, as fp32 (the scalar path below).
template <int KV>
__device__ __forceinline__ float cache_element(const unsigned char* row, int e) {
  if (KV == kKvF16) return __half2float(reinterpret_cast<const __half*>(row)[e]);
  if (KV == kKvFp8) return e4m3_to_float(row[e]);
  if (KV == kKvInt8) return static_cast<float>(static_cast<signed char>(row[e]));
  return static_cast<float>(static_cast<int>(static_cast<uint32_t>(row[e >> 1]) << (28 - 4 * (e & 1))) >> 28);
}

// The keys [start, last] query row i sees.
__device__ __forceinline__ void key_range(const AttnParams& p, int i, int& start, int& last) {
  const unsigned long long pos = p.q_base + i;
  last = p.causal ? static_cast<int>(pos >= static_cast<unsigned long long>(p.n) ? p.n - 1 : pos) : p.n - 1;
  start = 0;
  if (p.causal && p.window != 0 && pos + 1 > static_cast<unsigned long long>(p.window)) {
    const unsigned long long s = pos + 1 - p.window;
    start = s > static_cast<unsigned long long>(last) ? last : static_cast<int>(s);
  }
}

__device__ __forceinline__ float gated(float v, const float* gate, size_t at) {
  return gate != nullptr ? v / (1.0f + expf(-gate[at])) : v;
}

// grid: (kv_heads * row_tiles, splits).  Shared memory: the queries' two terms, one tile of keys and one of values in
// binary16 (rows of D elements, 16-byte chunk c of row r at c ^ (r & 7): ldmatrix and the stores are conflict-free),
// and for the narrower formats the next tiles' raw bytes, which arrive by cp.async while a tile is worked on (fp16
// tiles arrive in place).  A warp owns 16 rows: 64 scores and D outputs per row in registers.
template <int KV, int D>
__global__ void __launch_bounds__(kTileThreads, 1) attention_tile_kernel(const AttnTileParams tp) {
  using S = TileShape<KV, D>;
  constexpr bool kScaled = KV >= kKvFp8;
  constexpr int kPitch = D * 2;  // bytes of a binary16 row
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* const q_s = smem;  // [2 terms][128 rows][D]
  unsigned char* const k_s = q_s + S::kQBytes;
  unsigned char* const v_s = k_s + S::kTileBytes;
  unsigned char* const k_raw = v_s + S::kTileBytes;
  unsigned char* const v_raw = k_raw + S::kRawBytes;
  float* const row_f = reinterpret_cast<float*>(v_raw + S::kRawBytes);  // [128] score factor of a row
  float* const sc_s = row_f + kTileRows;                                 // [2 buffers][k, v][64] scales of a tile's keys
  float* const red = sc_s + 4 * kTileKeys;                               // [8]
  const AttnParams& p = tp.a;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, group = tp.group;
  const int kv = blockIdx.x % p.kv_heads, rt = tp.row_tiles - 1 - static_cast<int>(blockIdx.x) / p.kv_heads, split = blockIdx.y;
  const int rows_all = p.m * group, row0 = rt * kTileRows;
  const int rows = min(kTileRows, rows_all - row0);
  int first, last, unused;
  key_range(p, row0 / group, first, unused);
  key_range(p, (row0 + rows - 1) / group, unused, last);
  const int c0 = first + split * tp.tiles_per_split * kTileKeys;
  const int c1 = static_cast<int>(min(static_cast<long long>(last) + 1, static_cast<long long>(c0) + static_cast<long long>(tp.tiles_per_split) * kTileKeys));
  const int tiles = c1 > c0 ? (c1 - c0 + kTileKeys - 1) / kTileKeys : 0;
  const unsigned char* kbase = static_cast<const unsigned char*>(p.k) + static_cast<size_t>(kv) * S::kRowBytes;
  const unsigned char* vbase = static_cast<const unsigned char*>(p.v) + static_cast<size_t>(kv) * S::kRowBytes;
  const size_t row_bytes = static_cast<size_t>(p.kv_heads) * S::kRowBytes;
  bool bad = false;  // an infinity or NaN among what this thread has seen

  auto load_tile = [&](const unsigned char* base, unsigned char* raw, unsigned char* tile, int t) {
    if (t < tiles) {
#pragma unroll
      for (int it = 0; it < S::kPieces; ++it) {
        const int idx = tid + it * kTileThreads, r = idx / S::kPiecesPerRow, c = idx % S::kPiecesPerRow;
        const int j = min(c0 + t * kTileKeys + r, c1 - 1);
        const uint32_t dst = KV == kKvF16 ? smem_addr(tile + r * kPitch + ((c ^ (r & 7)) << 4)) : smem_addr(raw + idx * 16);
        cp_async16(dst, base + j * row_bytes + c * 16);
      }
    }
    cp_async_commit();
  };
  // the thread's own raw pieces -> binary16 (fp16 tiles only look for what is not finite)
  auto convert_tile = [&](unsigned char* raw, unsigned char* tile) {
#pragma unroll
    for (int it = 0; it < S::kPieces; ++it) {
      const int idx = tid + it * kTileThreads, r = idx / S::kPiecesPerRow, c = idx % S::kPiecesPerRow;
      if constexpr (KV == kKvF16) {
        const uint4 x = *reinterpret_cast<const uint4*>(tile + r * kPitch + ((c ^ (r & 7)) << 4));
        bad |= has_nonfinite_f16(x.x) || has_nonfinite_f16(x.y) || has_nonfinite_f16(x.z) || has_nonfinite_f16(x.w);
      } else {
        constexpr int kChunks = KV == kKvInt4 ? 4 : 2;  // 16-byte chunks of binary16 a piece becomes
        const uint4 x = *reinterpret_cast<const uint4*>(raw + idx * 16);
        const uint32_t w[4] = {x.x, x.y, x.z, x.w};
        uint32_t h[4][KV == kKvInt4 ? 4 : 2];
#pragma unroll
        for (int i = 0; i < 4; ++i) bad |= expand_word<KV>(w[i], h[i]);
#pragma unroll
        for (int o = 0; o < kChunks; ++o) {
          const uint4 y = KV == kKvInt4 ? make_uint4(h[o][0], h[o][1], h[o][2 % (kChunks)], h[o][3 % (kChunks)])
                                        : make_uint4(h[2 * (o & 1)][0], h[2 * (o & 1)][1], h[2 * (o & 1) + 1][0], h[2 * (o & 1) + 1][1]);
          *reinterpret_cast<uint4*>(tile + r * kPitch + (((c * kChunks + o) ^ (r & 7)) << 4)) = y;
        }
      }
    }
  };
  // scale of key tid % 64 of tile t (threads 0..63 the keys', 64..127 the values')
  auto load_scale = [&](int t) -> float {
    if (!kScaled || tid >= 2 * kTileKeys || t >= tiles) return 1.0f;
    const int j = min(c0 + t * kTileKeys + (tid & (kTileKeys - 1)), c1 - 1);
    return __ldg((tid < kTileKeys ? p.ks : p.vs) + j);
  };
  load_tile(kbase, k_raw, k_s, 0);
  load_tile(vbase, v_raw, v_s, 0);

  // value scales enter the weights relative to the chunk's largest one
  float v_norm = static_cast<float>(1 << kWeightBits), v_unit = 1.0f / static_cast<float>(1 << kWeightBits);
  if (kScaled) {
    float top = 0.0f;
#pragma unroll 4
    for (int j = c0 + tid; j < c1; j += kTileThreads) {
      const float s = fabsf(__ldg(p.vs + j));
      bad |= !(s <= 3.402823466e38f);
      top = fmaxf(top, s);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
    if (lane == 0) red[warp] = top;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kTileThreads / 32; ++w) top = fmaxf(top, red[w]);
    int e = static_cast<int>((__float_as_uint(top) >> 23) & 0xFFu) - 127;
    e = max(-100, min(100, e));
    if (top == 0.0f) e = 0;
    v_norm = __uint_as_float(static_cast<uint32_t>(127 + kWeightBits - e) << 23);
    v_unit = __uint_as_float(static_cast<uint32_t>(127 - kWeightBits + e) << 23);
  }
  // queries, in base-2 exponents: each row scaled by a power of two to [2^13, 2^14), two binary16 terms.  A score's
  // factor is then its key's scale times a power of two.
  const float q_scale = kLog2e / sqrtf(static_cast<float>(D));
  constexpr int kRowsAtOnce = 4;  // loads in flight together
  for (int rr = 0; rr < 16; rr += kRowsAtOnce) {
    float4 x[kRowsAtOnce][D / 128];
    float top[kRowsAtOnce];
#pragma unroll
    for (int u = 0; u < kRowsAtOnce; ++u) {
      const int r = warp * 16 + rr + u, i = (row0 + r) / group, g = (row0 + r) - i * group;
      const float* src = p.q + ((p.row_base + i) * p.heads + static_cast<size_t>(kv) * group + g) * D + lane * 4;
#pragma unroll
      for (int it = 0; it < D / 128; ++it)
        x[u][it] = r < rows ? __ldg(reinterpret_cast<const float4*>(src + it * 128)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
#pragma unroll
    for (int u = 0; u < kRowsAtOnce; ++u) {
      top[u] = 0.0f;
#pragma unroll
      for (int it = 0; it < D / 128; ++it) {
        float4& y = x[u][it];
        y = make_float4(y.x * q_scale, y.y * q_scale, y.z * q_scale, y.w * q_scale);
        bad |= !(fabsf(y.x) <= 3.402823466e38f) || !(fabsf(y.y) <= 3.402823466e38f) || !(fabsf(y.z) <= 3.402823466e38f) ||
               !(fabsf(y.w) <= 3.402823466e38f);
        top[u] = fmaxf(top[u], fmaxf(fmaxf(fabsf(y.x), fabsf(y.y)), fmaxf(fabsf(y.z), fabsf(y.w))));
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
      for (int u = 0; u < kRowsAtOnce; ++u) top[u] = fmaxf(top[u], __shfl_xor_sync(0xFFFFFFFFu, top[u], o));
#pragma unroll
    for (int u = 0; u < kRowsAtOnce; ++u) {
      const int r = warp * 16 + rr + u;
      int e = static_cast<int>((__float_as_uint(top[u]) >> 23) & 0xFFu) - 127 - 13;
      e = max(-110, min(114, e));
      if (top[u] == 0.0f) e = 0;
      const float up = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
      if (lane == 0) row_f[r] = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
#pragma unroll
      for (int it = 0; it < D / 128; ++it) {
        uint2 hi, lo;
        split_half2(x[u][it].x * up, x[u][it].y * up, hi.x, lo.x);
        split_half2(x[u][it].z * up, x[u][it].w * up, hi.y, lo.y);
        const int chunk = it * 16 + (lane >> 1), at = r * kPitch + ((chunk ^ (r & 7)) << 4) + (lane & 1) * 8;
        *reinterpret_cast<uint2*>(q_s + at) = hi;
        *reinterpret_cast<uint2*>(q_s + S::kQBytes / 2 + at) = lo;
      }
    }
  }
  if (kScaled) {
    const float s = load_scale(0);
    bad |= !(fabsf(s) <= 3.402823466e38f);
    if (tid < 2 * kTileKeys) sc_s[tid] = tid < kTileKeys ? s : s * v_norm;
  }
  if (KV != kKvF16) {
    cp_async_wait<1>();
    convert_tile(k_raw, k_s);
    load_tile(kbase, k_raw, k_s, 1);
    cp_async_wait<1>();
    convert_tile(v_raw, v_s);
    load_tile(vbase, v_raw, v_s, 1);
  } else {
    cp_async_wait<0>();
    convert_tile(k_raw, k_s);
    convert_tile(v_raw, v_s);
  }

  // a thread's two rows (of the m16n8 accumulators): warp * 16 + lane / 4 and + 8
  const int r_lo = warp * 16 + (lane >> 2);
  int start[2], stop[2];  // the keys of the row inside this chunk: start <= j < stop
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    int s = 0, l = -1;
    if (r_lo + 8 * u < rows) key_range(p, (row0 + r_lo + 8 * u) / group, s, l);
    start[u] = s;
    stop[u] = min(l + 1, c1);
  }
  const bool active = warp * 16 < rows;
  float o[D / 8][4];
#pragma unroll
  for (int n = 0; n < D / 8; ++n) o[n][0] = o[n][1] = o[n][2] = o[n][3] = 0.0f;
  float mx[2] = {kNoKey, kNoKey}, sum[2] = {0.0f, 0.0f};
  const uint32_t q_addr = smem_addr(q_s) + (warp * 16 + (lane & 15)) * kPitch;
  const uint32_t k_addr = smem_addr(k_s) + ((lane & 7) + ((lane >> 4) << 3)) * kPitch;
  const uint32_t v_addr = smem_addr(v_s) + (lane & 15) * kPitch;
  const uint32_t q_x = ((lane >> 4) ^ (lane & 7)) << 4, k_x = (((lane >> 3) & 1) ^ (lane & 7)) << 4, v_x = q_x;
  bool any_bad = __syncthreads_or(bad) != 0;

  for (int t = 0; t < tiles && !any_bad; ++t) {
    const int j0 = c0 + t * kTileKeys;
    const float next_scale = load_scale(t + 1);
    float s[kTileKeys / 8][4];
#pragma unroll
    for (int n = 0; n < kTileKeys / 8; ++n) s[n][0] = s[n][1] = s[n][2] = s[n][3] = 0.0f;
    if (active) {
#pragma unroll 4
      for (int k4 = 0; k4 < D / 16 / kScoreChain; ++k4) {
        float part[kTileKeys / 8][4];
#pragma unroll
        for (int n = 0; n < kTileKeys / 8; ++n) part[n][0] = part[n][1] = part[n][2] = part[n][3] = 0.0f;
#pragma unroll
        for (int k1 = 0; k1 < kScoreChain; ++k1) {
          const int kk = k4 * kScoreChain + k1;
          uint32_t ah[4], al[4], b[kTileKeys / 16][4];
          ldmatrix4(ah, q_addr + ((kk * 32) ^ q_x));
          ldmatrix4(al, q_addr + S::kQBytes / 2 + ((kk * 32) ^ q_x));
#pragma unroll
          for (int n = 0; n < kTileKeys / 16; ++n) ldmatrix4(b[n], k_addr + n * 16 * kPitch + ((kk * 32) ^ k_x));
#pragma unroll
          for (int n = 0; n < kTileKeys / 16; ++n) {
            mma_f16(part[2 * n], al, b[n][0], b[n][1]);
            mma_f16(part[2 * n + 1], al, b[n][2], b[n][3]);
          }
#pragma unroll
          for (int n = 0; n < kTileKeys / 16; ++n) {
            mma_f16(part[2 * n], ah, b[n][0], b[n][1]);
            mma_f16(part[2 * n + 1], ah, b[n][2], b[n][3]);
          }
        }
#pragma unroll
        for (int n = 0; n < kTileKeys / 8; ++n)
#pragma unroll
          for (int c = 0; c < 4; ++c) s[n][c] += part[n][c];
      }
    }
    if (KV == kKvF16) cp_async_wait<0>();  // this tile's values (they were asked for after the tile before)
    if (KV == kKvF16 && t > 0) convert_tile(v_raw, v_s);
    __syncthreads();  // everybody is done with the keys; the values are there
    if (KV != kKvF16) {
      cp_async_wait<1>();
      if (t + 1 < tiles) convert_tile(k_raw, k_s);
      load_tile(kbase, k_raw, k_s, t + 2);
    } else {
      load_tile(kbase, k_raw, k_s, t + 1);
    }
    const float* ksc = sc_s + (t & 1) * 2 * kTileKeys;
    const float* vsc = ksc + kTileKeys;
    if (active) {
      const float rf[2] = {row_f[r_lo], row_f[r_lo + 8]};
      float top[2] = {kNoKey, kNoKey};
#pragma unroll
      for (int n = 0; n < kTileKeys / 8; ++n) {
        const int key = n * 8 + (lane & 3) * 2;
        const float2 f = kScaled ? *reinterpret_cast<const float2*>(ksc + key) : make_float2(1.0f, 1.0f);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const int j = j0 + key + (c & 1);
          const float v = s[n][c] * (rf[c >> 1] * ((c & 1) ? f.y : f.x));
          s[n][c] = (j >= start[c >> 1] && j < stop[c >> 1]) ? v : kNoKey;
          top[c >> 1] = fmaxf(top[c >> 1], s[n][c]);
        }
      }
      float corr[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        top[u] = fmaxf(top[u], __shfl_xor_sync(0xFFFFFFFFu, top[u], 1));
        top[u] = fmaxf(top[u], __shfl_xor_sync(0xFFFFFFFFu, top[u], 2));
        const float now = fmaxf(mx[u], top[u]);
        corr[u] = exp2f(mx[u] - now);  // 1 while the row has had no key (kNoKey - kNoKey)
        mx[u] = now;
        sum[u] *= corr[u];
      }
      if (__any_sync(0xFFFFFFFFu, corr[0] != 1.0f || corr[1] != 1.0f)) {
#pragma unroll
        for (int n = 0; n < D / 8; ++n) o[n][0] *= corr[0], o[n][1] *= corr[0], o[n][2] *= corr[1], o[n][3] *= corr[1];
      }
      float tile_sum[2] = {0.0f, 0.0f};  // added to the running sum as one: fewer roundings at its magnitude
#pragma unroll
      for (int n = 0; n < kTileKeys / 8; ++n) {
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          s[n][c] = s[n][c] == kNoKey ? 0.0f : exp2f(s[n][c] - mx[c >> 1]);
          tile_sum[c >> 1] += s[n][c];
        }
      }
      sum[0] += tile_sum[0], sum[1] += tile_sum[1];
      uint32_t ph[kTileKeys / 16][4], pl[kTileKeys / 16][4];
#pragma unroll
      for (int kk = 0; kk < kTileKeys / 16; ++kk) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int n = 2 * kk + h;
          const float2 f = kScaled ? *reinterpret_cast<const float2*>(vsc + n * 8 + (lane & 3) * 2) : make_float2(v_norm, v_norm);
          split_half2(s[n][0] * f.x, s[n][1] * f.y, ph[kk][2 * h], pl[kk][2 * h]);
          split_half2(s[n][2] * f.x, s[n][3] * f.y, ph[kk][2 * h + 1], pl[kk][2 * h + 1]);
        }
      }
#pragma unroll
      for (int k2 = 0; k2 < kTileKeys / 16 / kValueChain; ++k2) {
#pragma unroll
        for (int n = 0; n < D / 16; ++n) {
          float part[2][4] = {};
#pragma unroll
          for (int k1 = 0; k1 < kValueChain; ++k1) {
            const int kk = k2 * kValueChain + k1;
            uint32_t b[4];
            ldmatrix4_trans(b, v_addr + kk * 16 * kPitch + ((n * 32) ^ v_x));
            mma_f16(part[0], pl[kk], b[0], b[1]);
            mma_f16(part[1], pl[kk], b[2], b[3]);
            mma_f16(part[0], ph[kk], b[0], b[1]);
            mma_f16(part[1], ph[kk], b[2], b[3]);
          }
#pragma unroll
          for (int c = 0; c < 4; ++c) o[2 * n][c] += part[0][c], o[2 * n + 1][c] += part[1][c];
        }
      }
    }
    if (kScaled && tid < 2 * kTileKeys) {
      bad |= !(fabsf(next_scale) <= 3.402823466e38f);
      sc_s[((t + 1) & 1) * 2 * kTileKeys + tid] = tid < kTileKeys ? next_scale : next_scale * v_norm;
    }
    if (KV == kKvF16) {
      cp_async_wait<0>();
      if (t + 1 < tiles) convert_tile(k_raw, k_s);
    }
    any_bad = __syncthreads_or(bad) != 0;  // everybody is done with the values; the next keys are there
    if (KV != kKvF16) {
      cp_async_wait<1>();
      if (t + 1 < tiles) convert_tile(v_raw, v_s);
      load_tile(vbase, v_raw, v_s, t + 2);
    } else {
      load_tile(vbase, v_raw, v_s, t + 1);
    }
  }
  cp_async_wait<0>();

  const size_t chunk_stride = static_cast<size_t>(p.splits);
  if (any_bad) {
    // Infinities or NaN somewhere in the chunk: a two-term product of them is not the product, and a masked key's
    // zero weight would not mask them.  The whole chunk again, a warp per row and key by key in fp32.
    for (int r = warp; r < rows; r += kTileThreads / 32) {
      const int i = (row0 + r) / group, g = (row0 + r) - i * group;
      const size_t head_row = (p.row_base + i) * p.heads + static_cast<size_t>(kv) * group + g;
      int s0, l0;
      key_range(p, i, s0, l0);
      float x[D / 32], acc[D / 32];
#pragma unroll
      for (int e = 0; e < D / 32; ++e) x[e] = p.q[head_row * D + e * 32 + lane] * (kLog2e / sqrtf(static_cast<float>(D))), acc[e] = 0.0f;
      float top = kNoKey, total = 0.0f;
      for (int j = max(s0, c0); j < min(l0 + 1, c1); ++j) {
        const unsigned char *kr = kbase + j * row_bytes, *vr = vbase + j * row_bytes;
        float dot = 0.0f;
#pragma unroll
        for (int e = 0; e < D / 32; ++e) dot = fmaf(x[e], cache_element<KV>(kr, e * 32 + lane), dot);
        const float sc = warp_sum(dot) * (kScaled ? p.ks[j] : 1.0f);
        if (sc > top) {
          const float corr = exp2f(top - sc);
          total *= corr;
#pragma unroll
          for (int e = 0; e < D / 32; ++e) acc[e] *= corr;
          top = sc;
        }
        const float w = exp2f(sc - top);
        total += w;
#pragma unroll
        for (int e = 0; e < D / 32; ++e) acc[e] = fmaf(w * (kScaled ? p.vs[j] : 1.0f), cache_element<KV>(vr, e * 32 + lane), acc[e]);
      }
      const size_t at = head_row * D;
      const size_t part = (static_cast<size_t>(i) * p.heads + static_cast<size_t>(kv) * group + g) * chunk_stride + split;
#pragma unroll
      for (int e = 0; e < D / 32; ++e) {
        if (tp.out != nullptr) tp.out[at + e * 32 + lane] = gated(acc[e] / total, tp.gate, at + e * 32 + lane);
        else p.pacc[part * D + e * 32 + lane] = acc[e];
      }
      if (tp.out == nullptr && lane == 0) {
        p.pmax[part] = top == kNoKey && total == 0.0f ? kNullMax : top * kLn2;
        p.psum[part] = total;
      }
    }
    return;
  }
  if (!active) return;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    sum[u] += __shfl_xor_sync(0xFFFFFFFFu, sum[u], 1);
    sum[u] += __shfl_xor_sync(0xFFFFFFFFu, sum[u], 2);
    const int r = r_lo + 8 * u;
    if (r >= rows) continue;
    const int i = (row0 + r) / group, g = (row0 + r) - i * group;
    const size_t head = static_cast<size_t>(kv) * group + g;
    if (tp.out != nullptr) {
      const size_t at = ((p.row_base + i) * p.heads + head) * D + (lane & 3) * 2;
      const float f = v_unit / sum[u];
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
        *reinterpret_cast<float2*>(tp.out + at + n * 8) =
            make_float2(gated(o[n][2 * u] * f, tp.gate, at + n * 8), gated(o[n][2 * u + 1] * f, tp.gate, at + n * 8 + 1));
    } else {
      const size_t part = (static_cast<size_t>(i) * p.heads + head) * chunk_stride + split;
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
        *reinterpret_cast<float2*>(p.pacc + part * D + n * 8 + (lane & 3) * 2) = make_float2(o[n][2 * u] * v_unit, o[n][2 * u + 1] * v_unit);
      if ((lane & 3) == 0) {
        p.pmax[part] = mx[u] == kNoKey ? kNullMax : mx[u] * kLn2;
        p.psum[part] = sum[u];
      }
    }
  }
}

// The chunks of a (row, head): a thread per four elements, chunks in order (attention_combine's arithmetic; that
// kernel spends a CTA on 64 elements of one row, which costs more than the reads once there are thousands of rows).
__global__ void __launch_bounds__(256)
attention_merge_kernel(const float* __restrict__ pacc, const float* __restrict__ pmax, const float* __restrict__ psum,
                       float* __restrict__ out, const float* __restrict__ gate, int dim4, int splits, size_t total,
                       size_t out_base) {
  const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const size_t row = t / dim4, e = t - row * dim4, base = row * splits;
  float top = kNullMax, den = 0.0f;
  for (int s = 0; s < splits; ++s) top = fmaxf(top, pmax[base + s]);
  float4 num = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float w = expf(pmax[base + s] - top);
    const float4 x = reinterpret_cast<const float4*>(pacc)[(base + s) * dim4 + e];
    den = fmaf(w, psum[base + s], den);
    num = make_float4(fmaf(w, x.x, num.x), fmaf(w, x.y, num.y), fmaf(w, x.z, num.z), fmaf(w, x.w, num.w));
  }
  const size_t at = (out_base + t) * 4;
  *reinterpret_cast<float4*>(out + at) = make_float4(gated(num.x / den, gate, at), gated(num.y / den, gate, at + 1),
                                                     gated(num.z / den, gate, at + 2), gated(num.w / den, gate, at + 3));
}

template <int KV, int D>
int launch_tile(const AttnTileParams& tp, cudaStream_t st) {
  auto kernel = attention_tile_kernel<KV, D>;
  static_assert(TileShape<KV, D>::kSmem <= 227 * 1024, "shared memory of a CTA");
  if (int rc = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), TileShape<KV, D>::kSmem)) return rc;
  const dim3 grid(static_cast<unsigned>(tp.a.kv_heads * tp.row_tiles), static_cast<unsigned>(tp.a.splits));
  kernel<<<grid, kTileThreads, TileShape<KV, D>::kSmem, st>>>(tp);
  return check_launch();
}

template <int KV>
int launch_tile_d(const AttnTileParams& tp, cudaStream_t st) {
  return tp.a.head_dim == 256 ? launch_tile<KV, 256>(tp, st) : launch_tile<KV, 128>(tp, st);
}

bool overlap(const void* a, size_t an, const void* b, size_t bn) {
  const auto *x = static_cast<const unsigned char*>(a), *y = static_cast<const unsigned char*>(b);
  return x < y + bn && y < x + an;
}
bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

}  // namespace

int attention_tile(int kvkind, AttnParams p, float* out, const float* gate, cudaStream_t st) {
  const int group = p.heads / p.kv_heads;
  const long rows = static_cast<long>(p.m) * group;
  // keys a row tile walks over: the window of its first row to the position of its last
  long span = p.n;
  if (p.causal && p.window != 0) span = span < p.window + kTileRows / group + 1 ? span : p.window + kTileRows / group + 1;
  if (p.causal && p.q_base + static_cast<unsigned long long>(p.m) < static_cast<unsigned long long>(span))
    span = static_cast<long>(p.q_base) + p.m;
  // Below a few rows a CTA's 128-row tile is mostly empty, and a short call is over before the tile's start has paid
  // off: measured (FP8, chunk kernel -> here) 8 rows x 200 keys 18 -> 20 us, 16 x 300 22.8 -> 23.8, 8 x 1024 28.9 -> 22.8,
  // 4 x 4096 45 -> 30, 16 x 4096 150 -> 36 (24 heads over 4 of 256); 2 rows x 4096 29 -> 29.
  // 16-byte pieces of q, the cache and the output; the chunk kernel takes what is not aligned.
  if (kvkind == kKvF32 || p.m < 4 || static_cast<double>(p.m) * span * p.kv_heads * p.head_dim < 8.0e6 || !aligned16(p.q) ||
      !aligned16(p.k) || !aligned16(p.v) || !aligned16(out))
    return kUnsupportedFeature;
  // With one chunk the result is written while other CTAs still read their queries and the cache.  In place over q is
  // fine (a CTA reads its own rows before it writes them); any other overlap stays with the chunk kernel, whose merge
  // starts when everything has been read.
  const size_t out_bytes = static_cast<size_t>(p.m) * p.heads * p.head_dim * 4;
  const size_t cache_bytes = static_cast<size_t>(p.n) * p.kv_heads * p.head_dim * (kvkind == kKvF16 ? 4 : kvkind == kKvInt4 ? 1 : 2) / 2;
  const float *rows_q = p.q + p.row_base * p.heads * p.head_dim, *rows_out = out + p.row_base * p.heads * p.head_dim;
  const size_t scale_bytes = kvkind == kKvF16 ? 0 : static_cast<size_t>(p.n) * 4;
  if ((rows_out != rows_q && overlap(rows_out, out_bytes, rows_q, out_bytes)) || overlap(rows_out, out_bytes, p.k, cache_bytes) ||
      overlap(rows_out, out_bytes, p.v, cache_bytes) ||
      (scale_bytes != 0 && (overlap(rows_out, out_bytes, p.ks, scale_bytes) || overlap(rows_out, out_bytes, p.vs, scale_bytes))) ||
      (gate != nullptr && overlap(rows_out, out_bytes, gate + p.row_base * p.heads * p.head_dim, out_bytes)))
    return kUnsupportedFeature;
  static const int sms = [] {
    int dev = 0, v = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    return v > 0 ? v : 148;
  }();
  const int row_tiles = static_cast<int>((rows + kTileRows - 1) / kTileRows);
  const long units = static_cast<long>(row_tiles) * p.kv_heads;
  const long tiles = (span + kTileKeys - 1) / kTileKeys;
  // Chunks of the key range: as many as make whole waves of CTAs, a CTA's start (queries, first tiles) counted as
  // two tiles and the merge of the chunks by its bytes.
  long best_splits = 1;
  double best = 0.0;
  const double merge_tile = static_cast<double>(p.m) * p.heads * p.head_dim * 8.0 / 5.0e12 / 4.5e-6;  // in tiles of 4.5 us
  for (long s = 1; s <= 64 && s <= tiles; ++s) {
    const long per = (tiles + s - 1) / s;
    if (s > 1 && (tiles + per - 1) / per != s) continue;  // chunks that would stay empty
    const double waves = static_cast<double>((units * s + sms - 1) / sms);
    const double cost = waves * (per + 2.0) + (s > 1 ? 1.0 + merge_tile * s : 0.0);
    if (s == 1 || cost < best) best = cost, best_splits = s;
  }
  AttnTileParams tp{};
  p.splits = static_cast<int>(best_splits);
  tp.group = group;
  tp.row_tiles = row_tiles;
  tp.tiles_per_split = static_cast<int>((tiles + best_splits - 1) / best_splits);
  if (best_splits > 1) {
    const size_t parts = static_cast<size_t>(p.m) * p.heads * best_splits;
    const size_t acc_bytes = parts * p.head_dim * 4, stat_bytes = (parts * 4 + 255) / 256 * 256;
    unsigned char* scratch = stream_scratch(st, acc_bytes + 2 * stat_bytes, 2);
    if (scratch != nullptr) {
      p.pacc = reinterpret_cast<float*>(scratch);
      p.pmax = reinterpret_cast<float*>(scratch + acc_bytes);
      p.psum = reinterpret_cast<float*>(scratch + acc_bytes + stat_bytes);
    } else {  // a capture before the first plain launch: no chunks
      p.splits = 1;
      tp.tiles_per_split = static_cast<int>(tiles);
    }
  }
  tp.a = p;
  tp.out = p.splits == 1 ? out : nullptr;
  tp.gate = gate;
  int rc;
  switch (kvkind) {
    case kKvF16: rc = launch_tile_d<kKvF16>(tp, st); break;
    case kKvFp8: rc = launch_tile_d<kKvFp8>(tp, st); break;
    case kKvInt4: rc = launch_tile_d<kKvInt4>(tp, st); break;
    default: rc = launch_tile_d<kKvInt8>(tp, st); break;
  }
  if (rc != kOk || p.splits == 1) return rc;
  const size_t total = static_cast<size_t>(p.m) * p.heads * p.head_dim / 4;
  attention_merge_kernel<<<static_cast<unsigned>((total + 255) / 256), 256, 0, st>>>(
      p.pacc, p.pmax, p.psum, out, gate, p.head_dim / 4, p.splits, total, p.row_base * p.heads * p.head_dim / 4);
  return check_launch();
}

}  // namespace tsr
