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
// 2^-38 below the row's largest weight of a tile.  Scales of quantised rows multiply the score and the weight in fp32, the
// latter before it is split: what a row does not see, or hardly weighs, takes nothing from it.  The
// MMA cuts off what falls below its accumulator instead of rounding (chains over 4096 keys came out 4e-6 off), and fp32 sums
// round at every step, so: the small terms have accumulators of their own, where what is cut off does not count; the leading
// terms of a score go through one MMA at a time, pairs of which are added to two sums, those of an output through four;
// factor and maximum meet a score in one fused multiply-add; fp16 elements, whose products with a leading term are longer
// than the accumulator, enter as their six leading bits and the rest.  Errors against 64 bits, the chunk kernel's in
// brackets (512 rows, 4096 keys, 24 heads of 256; int8 2048 keys, 4-bit 300 rows): FP8 2.6e-7 (3.0e-7), int8 2.3e-7 (2.8e-7),
// 4-bit 1.4e-7 (1.6e-7), fp16 2.16e-7 (2.19e-7).  With both terms in one accumulator, a single sum per score and a rounding
// before the maximum is taken off it was 3.8e-7, 3.7e-7, 2.2e-7 and 3.1e-7, 6 % (fp16 45 %) faster.
//
// Not built: the same on tcgen05, whose A operand can lie in tensor memory (weights without shared memory) and whose per-tile
// sums would be added to fp32 registers as here.  Open there: the leading terms of a score keep their accuracy for one MMA of 16
// elements, so every such product would be read back from tensor memory by itself.
// Bound: the tensor pipe as two warps a scheduler reach it with mma.sync (48 % busy, the rest fixed latencies and waits for the
// pipe): four MMAs where a plain product needs two (fp16: six).  512 rows over 4096
// keys, 24 heads of 256: FP8 423 us against the chunk kernel's 4470 (114 TFLOP/s of the contract's 48 GFLOP, 228 of the MMAs'),
// fp16 589 us against 4615.  255 registers a thread, 16 to 60 bytes spilled.
#include <cuda_fp16.h>

#include <atomic>

#include "attention.cuh"
#include "attention_plan.h"
#include "codec.cuh"
#include "launch.h"

namespace tsr {
namespace {

constexpr int kTileThreads = 256;
constexpr int kWeightBits = 14;  // a row's largest weight (times its key's value scale) is stored in [2^14, 2^15)
constexpr int kMinWeightExp = kWeightBits - 126;  // below, the power of two that takes it back would not be normal

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
  static constexpr int kSmem = kQBytes + 2 * kTileBytes + 2 * kRawBytes + kTileRows * 4 + 2 * 2 * kTileKeys * 4;
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
// The same from zero.
__device__ __forceinline__ void mma_f16_first(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
      : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
__device__ __forceinline__ __half2 u32_half2(uint32_t v) { return *reinterpret_cast<const __half2*>(&v); }
__device__ __forceinline__ uint32_t pack_half2(__half2 h) { return *reinterpret_cast<const uint32_t*>(&h); }
// (x, y) as binary16 and what binary16 lost of them
__device__ __forceinline__ void split_half2(float x, float y, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x, y);
  const float2 f = __half22float2(h);
  hi = pack_half2(h);
  lo = pack_half2(__floats2half2_rn(x - f.x, y - f.y));
}

// The same of the products x u and y v: one rounding, that of the second term.
__device__ __forceinline__ void split_product2(float x, float y, float u, float v, uint32_t& hi, uint32_t& lo) {
  const __half2 h = __floats2half2_rn(x * u, y * v);
  const float2 f = __half22float2(h);
  hi = pack_half2(h);
  lo = pack_half2(__floats2half2_rn(fmaf(x, u, -f.x), fmaf(y, v, -f.y)));
}
// Leaves the six leading significant bits of two elements in place and returns the rest, both exact.
__device__ __forceinline__ uint32_t split_elements(uint32_t& w) {
  const uint32_t top = w & 0xFFE0FFE0u, rest = pack_half2(__hsub2(u32_half2(w), u32_half2(top)));
  w = top;
  return rest;
}
// sum + rest += x without a rounding at the sum's magnitude
__device__ __forceinline__ void add_exact(float& sum, float& rest, float x) {
  const float t = __fadd_rn(sum, x), z = __fsub_rn(t, sum);
  rest = __fadd_rn(rest, __fadd_rn(__fsub_rn(sum, __fsub_rn(t, z)), __fsub_rn(x, z)));
  sum = t;
}
// The two together; an infinite or NaN sum as it is (its rest is a NaN).
__device__ __forceinline__ float with_rest(float sum, float rest) { return rest == rest ? sum + rest : sum; }
// Pairwise sums (for their latency): with roundings on the way, and rounded once.
template <int N>
__device__ __forceinline__ float tree_sum(const float (&v)[N]) {
  float s[N];
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = v[i];
#pragma unroll
  for (int half = N / 2; half > 0; half >>= 1)
#pragma unroll
    for (int i = 0; i < half; ++i) s[i] += s[i + half];
  return s[0];
}
template <int N>
__device__ __forceinline__ float exact_sum(const float (&v)[N]) {
  float s[N], rest = 0.0f;
#pragma unroll
  for (int i = 0; i < N; ++i) s[i] = v[i];
#pragma unroll
  for (int half = N / 2; half > 0; half >>= 1)
#pragma unroll
    for (int i = 0; i < half; ++i) add_exact(s[i], rest, s[i + half]);
  return with_rest(s[0], rest);
}

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

// The power of two that takes a row's largest weight `most` to [2^14, 2^15), and its inverse.
__device__ __forceinline__ void weight_unit(float most, float& up, float& unit) {
  const int e = max(kMinWeightExp, static_cast<int>(__float_as_uint(most) >> 23) - 127);
  up = __uint_as_float(static_cast<uint32_t>(127 + kWeightBits - e) << 23);
  unit = __uint_as_float(static_cast<uint32_t>(127 - kWeightBits + e) << 23);
}

// exp2 of a score less the row's maximum.  The maximum is rounded and the difference is not, so x can lie above 0, by as much
// as the scores' own error where they are beyond 2^24: a weight stays below 2 all the same.
__device__ __forceinline__ float weight_of(float x) { return exp2f(fminf(x, 1.0f)); }

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

// Rows [row0, row0 + rows) of kv head `kv` over keys [c0, c1), a warp per row and key by key in fp32: for chunks that hold
// infinities or NaN.  The result goes to `acc_s` / `top_s` (base-2 exponent) / `total_s` by row, or is `out` itself, or the
// partial of chunk `split`.
template <int KV, int D>
__device__ __noinline__ void scalar_rows(const AttnParams& p, int kv, int group, int row0, int rows, int c0, int c1, int split,
                                         int warp, int warps, float* out, const float* gate, float* acc_s, float* top_s, float* total_s) {
  constexpr bool kScaled = KV >= kKvFp8;
  constexpr int kRowBytes = D * kv_bits<KV>() / 8;
  const int lane = threadIdx.x & 31;
  const size_t row_bytes = static_cast<size_t>(p.kv_heads) * kRowBytes;
  const unsigned char* kbase = static_cast<const unsigned char*>(p.k) + static_cast<size_t>(kv) * kRowBytes;
  const unsigned char* vbase = static_cast<const unsigned char*>(p.v) + static_cast<size_t>(kv) * kRowBytes;
  for (int r = warp; r < rows; r += warps) {
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
    const size_t part = (static_cast<size_t>(i) * p.heads + static_cast<size_t>(kv) * group + g) * p.splits + split;
#pragma unroll
    for (int e = 0; e < D / 32; ++e) {
      if (acc_s != nullptr) acc_s[r * D + e * 32 + lane] = acc[e];
      else if (out != nullptr) out[at + e * 32 + lane] = gated(acc[e] / total, gate, at + e * 32 + lane);
      else p.pacc[part * D + e * 32 + lane] = acc[e];
    }
    if (acc_s != nullptr) {
      if (lane == 0) top_s[r] = top, total_s[r] = total;
    } else if (out == nullptr && lane == 0) {
      p.pmax[part] = top == kNoKey && total == 0.0f ? kNullMax : top * kLn2;
      p.psum[part] = total;
    }
  }
}

// grid: (kv_heads * row_tiles, splits).  Shared memory: the queries' two terms, one tile of keys and one of values in
// binary16 (rows of D elements, 16-byte chunk c of row r at c ^ (r & 7): ldmatrix and the stores are conflict-free),
// and for the narrower formats the next tiles' raw bytes, which arrive by cp.async while a tile is worked on (fp16
// tiles arrive in place).  A warp owns 16 rows: 64 scores and D outputs per row in registers.
template <int KV, int D>
__global__ void __launch_bounds__(kTileThreads, 1) attention_tile_kernel(const AttnTileParams tp) {
  using S = TileShape<KV, D>;
  constexpr bool kScaled = KV >= kKvFp8;
  constexpr bool kLongElements = KV == kKvF16;  // eleven significant bits
  constexpr int kPitch = D * 2;  // bytes of a binary16 row
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char* const q_s = smem;  // [2 terms][128 rows][D]
  unsigned char* const k_s = q_s + S::kQBytes;
  unsigned char* const v_s = k_s + S::kTileBytes;
  unsigned char* const k_raw = v_s + S::kTileBytes;
  unsigned char* const v_raw = k_raw + S::kRawBytes;
  float* const row_f = reinterpret_cast<float*>(v_raw + S::kRawBytes);  // [128] score factor of a row
  float* const sc_s = row_f + kTileRows;                                 // [2 buffers][k, v][64] scales of a tile's keys
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

  // queries: each row scaled by a power of two to [2^13, 2^14), two binary16 terms.  A score's factor (to a base-2 exponent)
  // is then its key's scale times a power of two; without key scales it has room for 1 / sqrt(D) too, which rounds the
  // elements otherwise.
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
        if (kScaled) y = make_float4(y.x * q_scale, y.y * q_scale, y.z * q_scale, y.w * q_scale);
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
      if (lane == 0) row_f[r] = __uint_as_float(static_cast<uint32_t>(127 + e) << 23) * (kScaled ? 1.0f : q_scale);
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
    if (tid < 2 * kTileKeys) sc_s[tid] = s;
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
  float mx[2] = {kNoKey, kNoKey}, sum[2] = {0.0f, 0.0f}, sum_rest[2] = {0.0f, 0.0f};
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
#pragma unroll
      for (int half = 0; half < 2; ++half) {  // 32 keys at a time: registers
        constexpr int kN = kTileKeys / 16;
        float low[kN][4] = {}, acc[2][kN][4] = {};
#pragma unroll 1
        for (int k4 = 0; k4 < D / 64; ++k4) {
          float first[kN][4];
#pragma unroll
          for (int k1 = 0; k1 < 4; ++k1) {
            const int kk = k4 * 4 + k1;
            uint32_t ah[4], al[4], b[kN / 2][4];
            ldmatrix4(ah, q_addr + ((kk * 32) ^ q_x));
            ldmatrix4(al, q_addr + S::kQBytes / 2 + ((kk * 32) ^ q_x));
#pragma unroll
            for (int n = 0; n < kN / 2; ++n) ldmatrix4(b[n], k_addr + (half * 2 + n) * 16 * kPitch + ((kk * 32) ^ k_x));
            float part[kN][4];
#pragma unroll
            for (int n = 0; n < kN; ++n) mma_f16(low[n], al, b[n / 2][2 * (n & 1)], b[n / 2][2 * (n & 1) + 1]);
            if constexpr (kLongElements) {
#pragma unroll
              for (int n = 0; n < kN; ++n) {
                const uint32_t r0 = split_elements(b[n / 2][2 * (n & 1)]), r1 = split_elements(b[n / 2][2 * (n & 1) + 1]);
                mma_f16(low[n], ah, r0, r1);
              }
            }
#pragma unroll
            for (int n = 0; n < kN; ++n) mma_f16_first(part[n], ah, b[n / 2][2 * (n & 1)], b[n / 2][2 * (n & 1) + 1]);
#pragma unroll
            for (int n = 0; n < kN; ++n)
#pragma unroll
              for (int c = 0; c < 4; ++c) {
                if (k1 % 2 == 0) first[n][c] = part[n][c];
                else acc[k1 / 2][n][c] += first[n][c] + part[n][c];
              }
          }
        }
#pragma unroll
        for (int n = 0; n < kN; ++n)
#pragma unroll
          for (int c = 0; c < 4; ++c) s[half * kN + n][c] = acc[0][n][c] + (acc[1][n][c] + low[n][c]);
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
          if (j >= start[c >> 1] && j < stop[c >> 1]) top[c >> 1] = fmaxf(top[c >> 1], s[n][c] * (rf[c >> 1] * ((c & 1) ? f.y : f.x)));
          else s[n][c] = kNoKey;
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
        sum[u] *= corr[u], sum_rest[u] *= corr[u];
      }
      if (__any_sync(0xFFFFFFFFu, corr[0] != 1.0f || corr[1] != 1.0f)) {
#pragma unroll
        for (int n = 0; n < D / 8; ++n) o[n][0] *= corr[0], o[n][1] *= corr[0], o[n][2] *= corr[1], o[n][3] *= corr[1];
      }
      float tile_sum[2] = {0.0f, 0.0f}, most[2] = {kScaled ? 0.0f : 1.0f, kScaled ? 0.0f : 1.0f}, up[2], unit[2];
#pragma unroll
      for (int n = 0; n < kTileKeys / 8; ++n) {
        const int key = n * 8 + (lane & 3) * 2;
        const float2 fk = kScaled ? *reinterpret_cast<const float2*>(ksc + key) : make_float2(1.0f, 1.0f);
        const float2 fv = kScaled ? *reinterpret_cast<const float2*>(vsc + key) : make_float2(1.0f, 1.0f);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float x = fmaf(s[n][c], rf[c >> 1] * ((c & 1) ? fk.y : fk.x), -mx[c >> 1]);
          s[n][c] = s[n][c] == kNoKey ? 0.0f : weight_of(x);
          tile_sum[c >> 1] += s[n][c];
          if (kScaled) most[c >> 1] = fmaxf(most[c >> 1], fabsf(s[n][c] * ((c & 1) ? fv.y : fv.x)));
        }
      }
      add_exact(sum[0], sum_rest[0], tile_sum[0]);
      add_exact(sum[1], sum_rest[1], tile_sum[1]);
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        if (kScaled) {
          most[u] = fmaxf(most[u], __shfl_xor_sync(0xFFFFFFFFu, most[u], 1));
          most[u] = fmaxf(most[u], __shfl_xor_sync(0xFFFFFFFFu, most[u], 2));
        }
        weight_unit(most[u], up[u], unit[u]);
      }
      uint32_t ph[kTileKeys / 16][4], pl[kTileKeys / 16][4];
#pragma unroll
      for (int kk = 0; kk < kTileKeys / 16; ++kk) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int n = 2 * kk + h;
          const float2 fv = kScaled ? *reinterpret_cast<const float2*>(vsc + n * 8 + (lane & 3) * 2) : make_float2(1.0f, 1.0f);
          split_product2(s[n][0] * up[0], s[n][1] * up[0], fv.x, fv.y, ph[kk][2 * h], pl[kk][2 * h]);
          split_product2(s[n][2] * up[1], s[n][3] * up[1], fv.x, fv.y, ph[kk][2 * h + 1], pl[kk][2 * h + 1]);
        }
      }
#pragma unroll
      for (int n = 0; n < D / 16; ++n) {
        float part[2][4], low[2][4];
#pragma unroll
        for (int kk = 0; kk < kTileKeys / 16; ++kk) {
          uint32_t b[4];
          ldmatrix4_trans(b, v_addr + kk * 16 * kPitch + ((n * 32) ^ v_x));
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if (kk == 0) mma_f16_first(low[h], pl[kk], b[2 * h], b[2 * h + 1]);
            else mma_f16(low[h], pl[kk], b[2 * h], b[2 * h + 1]);
          }
#pragma unroll
          for (int h = 0; h < 2; ++h) {
            if constexpr (kLongElements) {
              const uint32_t r0 = split_elements(b[2 * h]), r1 = split_elements(b[2 * h + 1]);
              mma_f16(low[h], ph[kk], r0, r1);
            }
            if (kk == 0) mma_f16_first(part[h], ph[kk], b[2 * h], b[2 * h + 1]);
            else mma_f16(part[h], ph[kk], b[2 * h], b[2 * h + 1]);
          }
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < 4; ++c) o[2 * n + h][c] = fmaf(part[h][c] + low[h][c], unit[c >> 1], o[2 * n + h][c]);
      }
    }
    if (kScaled && tid < 2 * kTileKeys) {
      bad |= !(fabsf(next_scale) <= 3.402823466e38f);
      sc_s[((t + 1) & 1) * 2 * kTileKeys + tid] = next_scale;
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
  if (any_bad) {  // a two-term product with an infinity or NaN is not the product, and a masked key's zero weight would not mask it
    scalar_rows<KV, D>(p, kv, group, row0, rows, c0, c1, split, warp, kTileThreads / 32, tp.out, tp.gate, nullptr, nullptr,
                         nullptr);
    return;
  }
  if (!active) return;
#pragma unroll
  for (int u = 0; u < 2; ++u) {
    sum[u] = with_rest(sum[u], sum_rest[u]);
    sum[u] += __shfl_xor_sync(0xFFFFFFFFu, sum[u], 1);
    sum[u] += __shfl_xor_sync(0xFFFFFFFFu, sum[u], 2);
    const int r = r_lo + 8 * u;
    if (r >= rows) continue;
    const int i = (row0 + r) / group, g = (row0 + r) - i * group;
    const size_t head = static_cast<size_t>(kv) * group + g;
    if (tp.out != nullptr) {
      const size_t at = ((p.row_base + i) * p.heads + head) * D + (lane & 3) * 2;
      const float f = 1.0f / sum[u];
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
        *reinterpret_cast<float2*>(tp.out + at + n * 8) =
            make_float2(gated(o[n][2 * u] * f, tp.gate, at + n * 8), gated(o[n][2 * u + 1] * f, tp.gate, at + n * 8 + 1));
    } else {
      const size_t part = (static_cast<size_t>(i) * p.heads + head) * chunk_stride + split;
#pragma unroll
      for (int n = 0; n < D / 8; ++n)
        *reinterpret_cast<float2*>(p.pacc + part * D + n * 8 + (lane & 3) * 2) = make_float2(o[n][2 * u], o[n][2 * u + 1]);
      if ((lane & 3) == 0) {
        p.pmax[part] = mx[u] == kNoKey ? kNullMax : mx[u] * kLn2;
        p.psum[part] = sum[u];
      }
    }
  }
}

// ---- few rows (a decoded token, drafted ones, a short prompt) ----
// The chunk kernel of attention.cu is bound by its instructions (about 1000 for four keys of a warp), and its chunks meet
// in a second launch; a row tile is mostly padding.  Here a cluster of up to sixteen CTAs takes one kv head and 8 NT
// (row, head) pairs over the whole key range: a CTA a chunk, a warp sixteen keys at a time, and the chunks meet through
// distributed shared memory.  More pairs are more clusters, as long as they all run at a time (few_ctas, few_rows_win).
// The products are S^T = K Q^T and O^T = V^T P^T, so that eight rows fill an MMA.  Keys and values go from global memory
// to MMA fragments in registers without shared memory, because the order of the elements along a contraction and of the
// output rows is free: lane t of a key's four reads 16-byte pieces t, t + 4, ... of its row, and the queries are laid out in
// that order; lane g of a value's eight reads the g-th eighth of its row.  The weights come out of the score MMA with keys
// along g and are turned by movmatrix.  Two terms per query element and weight and exact cache elements as above; the MMAs
// of four steps are added pairwise and the cluster's chunks without roundings.  One row of 24 heads over 4 of 256 and 4096 FP8
// keys 11.7 us (chunk kernel 15.2) at 2.2e-7 against 64 bits (2.9e-7).  Bound: latency (64 CTAs, two trips a warp) and the
// registers: 179 to 255 a thread, and with sixteen rows of 256 up to 436 bytes spilled.
constexpr int kFewWarps = 8, kFewKeys = 16;  // a warp's keys at a time

template <int KV, int D, int NT>
struct FewShape {
  static constexpr int kRows = 8 * NT, kRowBytes = D * kv_bits<KV>() / 8;
  static constexpr int kPiece = 128 / kv_bits<KV>();               // elements of a 16-byte piece
  static constexpr int kKeyPieces = kRowBytes / 64;                // of a key row, per lane
  static constexpr int kValueWords = kRowBytes / 32;               // 32-bit words of a value row, per lane
  static constexpr int kEighth = D / 8 + 2, kPitch = 8 * kEighth + 4;  // of a row's sums: 8-byte stores without conflicts
  static constexpr int kQBytes = 2 * kRows * D * 2, kAccBytes = kRows * D * 4;
  static constexpr int kSmem = kQBytes + kAccBytes + kFewWarps * kRows * (kPitch + 2) * 4 + 4 * kRows * 4;
};

__device__ __forceinline__ uint32_t transpose_8x8(uint32_t v) {
  uint32_t r;
  asm volatile("movmatrix.sync.aligned.m8n8.trans.b16 %0, %1;" : "=r"(r) : "r"(v));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
__device__ __forceinline__ uint32_t cluster_addr(uint32_t local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
  return r;
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}

// One element of the result from `chunks` (<= N) CTAs' maximum, sum of weights and sum at these shared-memory addresses.
template <int N>
__device__ __forceinline__ float merged_chunks(int chunks, uint32_t top_at, uint32_t total_at, uint32_t acc_at) {
  float tops[N], totals[N], accs[N], top = kNoKey;
#pragma unroll
  for (int c = 0; c < N; ++c) {
    tops[c] = kNoKey, totals[c] = accs[c] = 0.0f;
    if (c < chunks) {
      tops[c] = ld_cluster(cluster_addr(top_at, c));
      totals[c] = ld_cluster(cluster_addr(total_at, c));
      accs[c] = ld_cluster(cluster_addr(acc_at, c));
    }
  }
#pragma unroll
  for (int c = 0; c < N; ++c) top = fmaxf(top, tops[c]);
#pragma unroll
  for (int c = 0; c < N; ++c)
    if (c < chunks) {
      const float w = exp2f(tops[c] - top);
      accs[c] *= w, totals[c] *= w;
    }
  return exact_sum(accs) / exact_sum(totals);
}

// grid: (kv_heads * splits, row tiles) in clusters of (splits, 1)
template <int KV, int D, int NT>
__global__ void __launch_bounds__(kFewWarps * 32, 1) attention_few_kernel(const AttnParams p, int group, float* out, const float* gate) {
  using S = FewShape<KV, D, NT>;
  static_assert(kv_bits<KV>() <= 8, "formats with a scale per row");
  constexpr int kWordSteps = kv_bits<KV>() == 8 ? 1 : 2;  // k steps a 32-bit word of a key feeds
  constexpr int kPer = 32 / kv_bits<KV>();                // elements of a word
  constexpr int kGroup = 4;  // MMA pairs in flight: the second of a pair waits for the first
  static_assert(4 * S::kKeyPieces % (kGroup / kWordSteps) == 0 && S::kValueWords % (2 * kGroup / kPer) == 0, "whole groups");
  constexpr int kRows = S::kRows;
  extern __shared__ __align__(128) unsigned char smem[];
  uint32_t* const q_s = reinterpret_cast<uint32_t*>(smem);                 // [D / 16][NT][hi, lo][32 lanes][2]
  float* const acc_s = reinterpret_cast<float*>(smem + S::kQBytes);        // [rows][D], the CTA's sums
  float* const part = acc_s + kRows * D;                                   // [warps][rows][kPitch]
  float* const wmax = part + kFewWarps * kRows * S::kPitch;                // [warps][rows]
  float* const wsum = wmax + kFewWarps * kRows;
  float* const top_s = wsum + kFewWarps * kRows;                           // [rows], the CTA's
  float* const total_s = top_s + kRows;
  float* const row_f = total_s + kRows;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
  const int kv = blockIdx.x / p.splits, split = blockIdx.x - kv * p.splits;
  const int row0 = blockIdx.y * kRows, rows = min(kRows, p.m * group - row0);
  int first, last, unused;
  key_range(p, row0 / group, first, unused);
  key_range(p, (row0 + rows - 1) / group, unused, last);
  const int keys = last - first + 1, chunk = (keys + p.splits - 1) / p.splits;
  const int c0 = first + split * chunk, c1 = min(last + 1, c0 + chunk);
  const unsigned char* kbase = static_cast<const unsigned char*>(p.k) + static_cast<size_t>(kv) * S::kRowBytes;
  const unsigned char* vbase = static_cast<const unsigned char*>(p.v) + static_cast<size_t>(kv) * S::kRowBytes;
  const size_t row_bytes = static_cast<size_t>(p.kv_heads) * S::kRowBytes;
  bool bad = false;

  uint32_t kraw[2][S::kKeyPieces][4], vraw[4][S::kValueWords];
  float ksc[2], vsc[2];  // of keys base + g and base + 8 + g
  auto load_keys = [&](int base) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = min(base + h * 8 + g, c1 - 1);
      const unsigned char* row = kbase + j * row_bytes;
#pragma unroll
      for (int u = 0; u < S::kKeyPieces; ++u) {
        const uint4 x = __ldg(reinterpret_cast<const uint4*>(row + (u * 4 + t) * 16));
        kraw[h][u][0] = x.x, kraw[h][u][1] = x.y, kraw[h][u][2] = x.z, kraw[h][u][3] = x.w;
      }
      ksc[h] = __ldg(p.ks + j), vsc[h] = __ldg(p.vs + j);
    }
  };
  auto load_values = [&](int base) {
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int j = min(base + 2 * t + (u & 1) + 8 * (u >> 1), c1 - 1);
      const unsigned char* row = vbase + j * row_bytes + g * (S::kRowBytes / 8);
      if constexpr (S::kValueWords >= 4) {
#pragma unroll
        for (int x4 = 0; x4 < S::kValueWords / 4; ++x4) {
          const uint4 x = __ldg(reinterpret_cast<const uint4*>(row) + x4);
          vraw[u][4 * x4] = x.x, vraw[u][4 * x4 + 1] = x.y, vraw[u][4 * x4 + 2] = x.z, vraw[u][4 * x4 + 3] = x.w;
        }
      } else {
        const uint2 x = __ldg(reinterpret_cast<const uint2*>(row));
        vraw[u][0] = x.x, vraw[u][1] = x.y;
      }
    }
  };
  const int begin = c0 + warp * kFewKeys;
  if (begin < c1) {
    load_keys(begin);
    load_values(begin);
  }

  // queries in fragment order, scaled as in the tile kernel: a warp per row
  const float q_scale = kLog2e / sqrtf(static_cast<float>(D));
#pragma unroll
  for (int u = 0; u < NT; ++u) {
    const int r = u * 8 + warp, i = (row0 + r) / group, hd = (row0 + r) - i * group;
    const float* src = p.q + ((p.row_base + i) * p.heads + static_cast<size_t>(kv) * group + hd) * D + lane * 4;
    float4 x[D / 128];
    float top = 0.0f;
#pragma unroll
    for (int it = 0; it < D / 128; ++it) {
      float4 y = r < rows ? __ldg(reinterpret_cast<const float4*>(src + it * 128)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      y = make_float4(y.x * q_scale, y.y * q_scale, y.z * q_scale, y.w * q_scale);
      bad |= !(fabsf(y.x) <= 3.402823466e38f) || !(fabsf(y.y) <= 3.402823466e38f) || !(fabsf(y.z) <= 3.402823466e38f) ||
             !(fabsf(y.w) <= 3.402823466e38f);
      top = fmaxf(top, fmaxf(fmaxf(fabsf(y.x), fabsf(y.y)), fmaxf(fabsf(y.z), fabsf(y.w))));
      x[it] = y;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, o));
    int e = static_cast<int>((__float_as_uint(top) >> 23) & 0xFFu) - 127 - 13;
    e = max(-110, min(114, e));
    if (top == 0.0f) e = 0;
    const float upf = __uint_as_float(static_cast<uint32_t>(127 - e) << 23);
    if (lane == 0) row_f[r] = __uint_as_float(static_cast<uint32_t>(127 + e) << 23);
#pragma unroll
    for (int it = 0; it < D / 128; ++it) {
      // elements d .. d + 3 are one lane's four of a k step: piece j = d / (4 kPiece), lane (d / kPiece) % 4
      const int d = it * 128 + lane * 4, j = d / (4 * S::kPiece), tq = (d / S::kPiece) & 3, step = j * (S::kPiece / 4) + (d % S::kPiece) / 4;
      uint2 hi, lo;
      split_half2(x[it].x * upf, x[it].y * upf, hi.x, lo.x);
      split_half2(x[it].z * upf, x[it].w * upf, hi.y, lo.y);
      uint2* const dst = reinterpret_cast<uint2*>(q_s) + (step * NT + u) * 64 + warp * 4 + tq;
      dst[0] = hi, dst[32] = lo;
    }
  }
  __syncthreads();

  int start[NT][2], stop[NT][2];  // of rows 8 nt + 2t and + 1, the rows of this lane's scores and sums
  float rf[NT][2], mx[NT][2], sum[NT][2];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int r = nt * 8 + 2 * t + u;
      int s0 = 0, l0 = -1;
      if (r < rows) key_range(p, (row0 + r) / group, s0, l0);
      start[nt][u] = s0, stop[nt][u] = min(l0 + 1, c1);
      rf[nt][u] = row_f[r], mx[nt][u] = kNoKey, sum[nt][u] = 0.0f;
    }
  float o[NT][D / 16][4];
#pragma unroll
  for (int nt = 0; nt < NT; ++nt)
#pragma unroll
    for (int j = 0; j < D / 16; ++j) o[nt][j][0] = o[nt][j][1] = o[nt][j][2] = o[nt][j][3] = 0.0f;
  for (int base = begin; base < c1; base += kFewWarps * kFewKeys) {
    const bool more = base + kFewWarps * kFewKeys < c1;
    float s[NT][4];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) s[nt][0] = s[nt][1] = s[nt][2] = s[nt][3] = 0.0f;
#pragma unroll
    for (int w0 = 0; w0 < 4 * S::kKeyPieces; w0 += kGroup / kWordSteps) {
      uint32_t b[2][kGroup / kWordSteps][2 * kWordSteps];
      float pt[kGroup][NT][4];
#pragma unroll
      for (int x = 0; x < kGroup / kWordSteps; ++x) {
        bad |= expand_word<KV>(kraw[0][(w0 + x) / 4][(w0 + x) % 4], b[0][x]);
        bad |= expand_word<KV>(kraw[1][(w0 + x) / 4][(w0 + x) % 4], b[1][x]);
      }
#pragma unroll
      for (int lo = 1; lo >= 0; --lo)
#pragma unroll
        for (int x = 0; x < kGroup; ++x) {
          const int wd = x / kWordSteps, h = 2 * (x % kWordSteps);
          const uint32_t a[4] = {b[0][wd][h], b[1][wd][h], b[0][wd][h + 1], b[1][wd][h + 1]};
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            const uint2 f = *reinterpret_cast<const uint2*>(q_s + (((w0 * kWordSteps + x) * NT + nt) * 64 + lo * 32 + lane) * 2);
            if (lo) mma_f16_first(pt[x][nt], a, f.x, f.y);
            else mma_f16(pt[x][nt], a, f.x, f.y);
          }
        }
#pragma unroll
      for (int nt = 0; nt < NT; ++nt)
#pragma unroll
        for (int c = 0; c < 4; ++c) s[nt][c] += (pt[0][nt][c] + pt[1][nt][c]) + (pt[2][nt][c] + pt[3][nt][c]);
    }
    const float ks0 = ksc[0], ks1 = ksc[1], vs0 = vsc[0], vs1 = vsc[1];
    if (more) load_keys(base + kFewWarps * kFewKeys);
    bad |= !(fabsf(ks0) <= 3.402823466e38f) || !(fabsf(ks1) <= 3.402823466e38f) || !(fabsf(vs0) <= 3.402823466e38f) ||
           !(fabsf(vs1) <= 3.402823466e38f);
    float unit[NT][2];
    uint32_t ph[NT][2], pl[NT][2];
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) {
      float corr[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int j = base + g;
        const float f0 = rf[nt][u] * ks0, f1 = rf[nt][u] * ks1;
        const bool in0 = j >= start[nt][u] && j < stop[nt][u], in1 = j + 8 >= start[nt][u] && j + 8 < stop[nt][u];
        float top = fmaxf(in0 ? s[nt][u] * f0 : kNoKey, in1 ? s[nt][2 + u] * f1 : kNoKey);
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xFFFFFFFFu, top, x));
        const float now = fmaxf(mx[nt][u], top);
        corr[u] = exp2f(mx[nt][u] - now);
        mx[nt][u] = now;
        s[nt][u] = in0 ? weight_of(fmaf(s[nt][u], f0, -now)) : 0.0f;
        s[nt][2 + u] = in1 ? weight_of(fmaf(s[nt][2 + u], f1, -now)) : 0.0f;
        sum[nt][u] = fmaf(sum[nt][u], corr[u], s[nt][u] + s[nt][2 + u]);
      }
      if (__any_sync(0xFFFFFFFFu, corr[0] != 1.0f || corr[1] != 1.0f)) {
#pragma unroll
        for (int j = 0; j < D / 16; ++j)
          o[nt][j][0] *= corr[0], o[nt][j][1] *= corr[1], o[nt][j][2] *= corr[0], o[nt][j][3] *= corr[1];
      }
      float up[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        float most = fmaxf(fabsf(s[nt][u] * vs0), fabsf(s[nt][2 + u] * vs1));
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) most = fmaxf(most, __shfl_xor_sync(0xFFFFFFFFu, most, x));
        weight_unit(most, up[u], unit[nt][u]);
      }
      split_product2(s[nt][0] * up[0], s[nt][1] * up[1], vs0, vs0, ph[nt][0], pl[nt][0]);
      split_product2(s[nt][2] * up[0], s[nt][3] * up[1], vs1, vs1, ph[nt][1], pl[nt][1]);
      ph[nt][0] = transpose_8x8(ph[nt][0]), ph[nt][1] = transpose_8x8(ph[nt][1]);
      pl[nt][0] = transpose_8x8(pl[nt][0]), pl[nt][1] = transpose_8x8(pl[nt][1]);
    }
#pragma unroll
    for (int w0 = 0; w0 < S::kValueWords; w0 += 2 * kGroup / kPer) {
      uint32_t b[2][2 * kGroup];  // keys 2t, 2t + 1 of an element; keys 2t + 8, 2t + 9
#pragma unroll
      for (int wd = 0; wd < 2 * kGroup / kPer; ++wd)
#pragma unroll
        for (int half = 0; half < 2; ++half) {
          const uint32_t wa = vraw[2 * half][w0 + wd], wb = vraw[2 * half + 1][w0 + wd];
          uint32_t* const dst = b[half] + wd * kPer;
          if constexpr (kv_bits<KV>() == 8) {
            uint32_t x[2], y[2];
            bad |= expand_word<KV>(__byte_perm(wa, wb, 0x5140), x);
            bad |= expand_word<KV>(__byte_perm(wa, wb, 0x7362), y);
            dst[0] = x[0], dst[1] = x[1], dst[2] = y[0], dst[3] = y[1];
          } else {  // the two keys' nibbles of an element side by side
            uint32_t x[4], y[4];
            expand_word<KV>((wa & 0x0F0F0F0Fu) | ((wb & 0x0F0F0F0Fu) << 4), x);
            expand_word<KV>(((wa >> 4) & 0x0F0F0F0Fu) | (wb & 0xF0F0F0F0u), y);
#pragma unroll
            for (int x4 = 0; x4 < 4; ++x4) dst[2 * x4] = x[x4], dst[2 * x4 + 1] = y[x4];
          }
        }
      float pt[kGroup][NT][4];
#pragma unroll
      for (int lo = 1; lo >= 0; --lo)
#pragma unroll
        for (int x = 0; x < kGroup; ++x) {
          const uint32_t a[4] = {b[0][2 * x], b[0][2 * x + 1], b[1][2 * x], b[1][2 * x + 1]};
#pragma unroll
          for (int nt = 0; nt < NT; ++nt) {
            if (lo) mma_f16_first(pt[x][nt], a, pl[nt][0], pl[nt][1]);
            else mma_f16(pt[x][nt], a, ph[nt][0], ph[nt][1]);
          }
        }
#pragma unroll
      for (int x = 0; x < kGroup; ++x)
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            float& sum_o = o[nt][w0 * kPer / 2 + x][c];
            sum_o = fmaf(pt[x][nt][c], unit[nt][c & 1], sum_o);
          }
    }
    if (more) load_values(base + kFewWarps * kFewKeys);
  }
  if (__syncthreads_or(bad)) {
    scalar_rows<KV, D>(p, kv, group, row0, rows, c0, c1, split, warp, kFewWarps, nullptr, nullptr, acc_s, top_s, total_s);
  } else {
    // the warps meet: the CTA's max per row, every warp's share rescaled to it
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
#pragma unroll
        for (int x = 4; x < 32; x <<= 1) sum[nt][u] += __shfl_xor_sync(0xFFFFFFFFu, sum[nt][u], x);
        if (g == 0) wmax[warp * kRows + nt * 8 + 2 * t + u] = mx[nt][u];
      }
    __syncthreads();
#pragma unroll
    for (int nt = 0; nt < NT; ++nt)
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int r = nt * 8 + 2 * t + u;
        float top = wmax[r];
#pragma unroll
        for (int w = 1; w < kFewWarps; ++w) top = fmaxf(top, wmax[w * kRows + r]);
        const float f = exp2f(mx[nt][u] - top);  // 0 for a warp that had no key (1 when none had: its sums are 0)
        if (g == 0) wsum[warp * kRows + r] = sum[nt][u] * f;
        float* dst = part + (warp * kRows + r) * S::kPitch + g * S::kEighth;
#pragma unroll
        for (int j = 0; j < D / 16; ++j) *reinterpret_cast<float2*>(dst + 2 * j) = make_float2(o[nt][j][u] * f, o[nt][j][2 + u] * f);
      }
    __syncthreads();
    for (int x = tid; x < rows * D; x += kFewWarps * 32) {
      const int r = x / D, d = x - r * D;
      const float* src = part + r * S::kPitch + d / (D / 8) * S::kEighth + d % (D / 8);
      float v[kFewWarps];
#pragma unroll
      for (int w = 0; w < kFewWarps; ++w) v[w] = src[w * kRows * S::kPitch];
      acc_s[x] = tree_sum(v);
    }
    if (tid < rows) {
      float top = wmax[tid], v[kFewWarps];
#pragma unroll
      for (int w = 1; w < kFewWarps; ++w) top = fmaxf(top, wmax[w * kRows + tid]);
#pragma unroll
      for (int w = 0; w < kFewWarps; ++w) v[w] = wsum[w * kRows + tid];
      top_s[tid] = top, total_s[tid] = tree_sum(v);
    }
  }
  // the chunks meet: CTA `split` merges its share of the elements, all CTAs' values in flight
  cluster_sync();
  const int share = (rows * D + p.splits - 1) / p.splits;
  const int begin_x = split * share + tid, end_x = min(rows * D, (split + 1) * share);
  for (int x = begin_x; x < end_x; x += kFewWarps * 32) {
    const int r = x / D, d = x - r * D, i = (row0 + r) / group, hd = (row0 + r) - i * group;
    const uint32_t top_at = smem_addr(top_s + r), total_at = smem_addr(total_s + r), acc_at = smem_addr(acc_s + x);
    const float v = p.splits <= 4 ? merged_chunks<4>(p.splits, top_at, total_at, acc_at) : merged_chunks<kFewCluster>(p.splits, top_at, total_at, acc_at);
    const size_t at = ((p.row_base + i) * p.heads + static_cast<size_t>(kv) * group + hd) * D + d;
    out[at] = gated(v, gate, at);
  }
  cluster_sync();  // the others may still read this CTA's sums
}

// The chunks of a (row, head): a thread per four elements, chunks in order (that of attention_combine; its
// kernel spends a CTA on 64 elements of one row, which costs more than the reads once there are thousands of rows).
__global__ void __launch_bounds__(256)
attention_merge_kernel(const float* __restrict__ pacc, const float* __restrict__ pmax, const float* __restrict__ psum,
                       float* __restrict__ out, const float* __restrict__ gate, int dim4, int splits, size_t total,
                       size_t out_base) {
  const size_t t = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (t >= total) return;
  const size_t row = t / dim4, e = t - row * dim4, base = row * splits;
  float top = kNullMax, den = 0.0f, den_rest = 0.0f, num[4] = {}, rest[4] = {};
  for (int s = 0; s < splits; ++s) top = fmaxf(top, pmax[base + s]);
#pragma unroll 4
  for (int s = 0; s < splits; ++s) {
    const float w = expf(pmax[base + s] - top);
    const float4 x = reinterpret_cast<const float4*>(pacc)[(base + s) * dim4 + e];
    add_exact(den, den_rest, w * psum[base + s]);
    add_exact(num[0], rest[0], w * x.x), add_exact(num[1], rest[1], w * x.y);
    add_exact(num[2], rest[2], w * x.z), add_exact(num[3], rest[3], w * x.w);
  }
  den = with_rest(den, den_rest);
#pragma unroll
  for (int c = 0; c < 4; ++c) num[c] = with_rest(num[c], rest[c]);
  const size_t at = (out_base + t) * 4;
  *reinterpret_cast<float4*>(out + at) = make_float4(gated(num[0] / den, gate, at), gated(num[1] / den, gate, at + 1),
                                                     gated(num[2] / den, gate, at + 2), gated(num[3] / den, gate, at + 3));
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

bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <int KV, int D, int NT>
cudaLaunchConfig_t few_config(cudaLaunchAttribute* cluster, int ctas, dim3 grid, cudaStream_t st) {
  cluster->id = cudaLaunchAttributeClusterDimension;
  cluster->val.clusterDim.x = static_cast<unsigned>(ctas);
  cluster->val.clusterDim.y = cluster->val.clusterDim.z = 1;
  cudaLaunchConfig_t config{};
  config.gridDim = grid;
  config.blockDim = dim3(kFewWarps * 32);
  config.dynamicSmemBytes = FewShape<KV, D, NT>::kSmem;
  config.stream = st;
  config.attrs = cluster;
  config.numAttrs = 1;
  return config;
}

// Clusters of `ctas` CTAs (a power of two) that the device runs at a time: a cluster lies within a GPC, so a B200 holds few
// of sixteen, more than twice as many of eight.  0 where it takes none of that size (a partitioned GPU).
template <int KV, int D, int NT>
int few_resident(int dev, int ctas) {
  static std::atomic<int> known[64][5];  // the number plus one; 0: not asked
  int log = 0;
  while ((1 << log) < ctas) ++log;
  if (int v = known[dev][log].load(std::memory_order_relaxed)) return v - 1;
  const auto kernel = &attention_few_kernel<KV, D, NT>;
  cudaLaunchAttribute cluster;
  const cudaLaunchConfig_t config = few_config<KV, D, NT>(&cluster, ctas, dim3(static_cast<unsigned>(ctas)), nullptr);
  int clusters = 0;
  if ((ctas > 8 && cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) ||
      cudaOccupancyMaxActiveClusters(&clusters, kernel, &config) != cudaSuccess) {
    cudaGetLastError();
    clusters = 0;
  }
  known[dev][log].store(clusters + 1, std::memory_order_relaxed);
  return clusters;
}

template <int KV, int D, int NT>
int launch_few_nt(AttnParams p, long span, int group, float* out, const float* gate, cudaStream_t st) {
  using S = FewShape<KV, D, NT>;
  const auto kernel = &attention_few_kernel<KV, D, NT>;
  if (int rc = allow_dynamic_smem(reinterpret_cast<const void*>(kernel), S::kSmem)) return rc;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return kDeviceError;
  const int row_tiles = (p.m * group + S::kRows - 1) / S::kRows;
  bool one_wave;
  p.splits = few_ctas(span, static_cast<int64_t>(p.kv_heads) * row_tiles, [&](int ctas) { return few_resident<KV, D, NT>(dev, ctas); }, &one_wave);
  if (p.m >= 4 && aligned16(out) && !few_rows_win(span, p.splits, one_wave, D)) return kUnsupportedFeature;
  cudaLaunchAttribute cluster;
  const cudaLaunchConfig_t config =
      few_config<KV, D, NT>(&cluster, p.splits, dim3(static_cast<unsigned>(p.kv_heads * p.splits), static_cast<unsigned>(row_tiles)), st);
  if (cudaLaunchKernelEx(&config, kernel, p, group, out, gate) != cudaSuccess) return kDeviceError;
  return check_launch();
}

template <int KV>
int launch_few(const AttnParams& p, long span, int group, float* out, const float* gate, cudaStream_t st) {
  if (p.m * group <= 8)
    return p.head_dim == 256 ? launch_few_nt<KV, 256, 1>(p, span, group, out, gate, st) : launch_few_nt<KV, 128, 1>(p, span, group, out, gate, st);
  return p.head_dim == 256 ? launch_few_nt<KV, 256, 2>(p, span, group, out, gate, st) : launch_few_nt<KV, 128, 2>(p, span, group, out, gate, st);
}

bool overlap(const void* a, size_t an, const void* b, size_t bn) {
  const auto *x = static_cast<const unsigned char*>(a), *y = static_cast<const unsigned char*>(b);
  return x < y + bn && y < x + an;
}

// Whether the result may be written while other CTAs still read their queries and the cache.  In place over q is fine (a
// CTA or cluster reads its own rows before it writes them); any other overlap stays with the chunk kernel, whose merge
// starts when everything has been read.
bool writes_apart(int kvkind, const AttnParams& p, const float* out, const float* gate) {
  const size_t out_bytes = static_cast<size_t>(p.m) * p.heads * p.head_dim * 4;
  const size_t cache_bytes = static_cast<size_t>(p.n) * p.kv_heads * p.head_dim * (kvkind == kKvF16 ? 4 : kvkind == kKvInt4 ? 1 : 2) / 2;
  const float *rows_q = p.q + p.row_base * p.heads * p.head_dim, *rows_out = out + p.row_base * p.heads * p.head_dim;
  const size_t scale_bytes = kvkind == kKvF16 ? 0 : static_cast<size_t>(p.n) * 4;
  return !((rows_out != rows_q && overlap(rows_out, out_bytes, rows_q, out_bytes)) || overlap(rows_out, out_bytes, p.k, cache_bytes) ||
           overlap(rows_out, out_bytes, p.v, cache_bytes) ||
           (scale_bytes != 0 && (overlap(rows_out, out_bytes, p.ks, scale_bytes) || overlap(rows_out, out_bytes, p.vs, scale_bytes))) ||
           (gate != nullptr && overlap(rows_out, out_bytes, gate + p.row_base * p.heads * p.head_dim, out_bytes)));
}

}  // namespace

int attention_few(int kvkind, AttnParams p, float* out, const float* gate, cudaStream_t st) {
  const int group = p.heads / p.kv_heads;
  const long span = p.causal && p.window != 0 && p.window < p.n ? p.window : p.n;
  if (kvkind < kKvFp8 || !aligned16(p.q) || !aligned16(p.k) || !aligned16(p.v) || !writes_apart(kvkind, p, out, gate))
    return kUnsupportedFeature;
  switch (kvkind) {
    case kKvFp8: return launch_few<kKvFp8>(p, span, group, out, gate, st);
    case kKvInt8: return launch_few<kKvInt8>(p, span, group, out, gate, st);
    default: return launch_few<kKvInt4>(p, span, group, out, gate, st);
  }
}

int attention_tile(int kvkind, AttnParams p, float* out, const float* gate, cudaStream_t st) {
  const int group = p.heads / p.kv_heads;
  const long rows = static_cast<long>(p.m) * group;
  const long span = static_cast<long>(tile_span(p.m, p.n, p.q_base, p.window, p.causal != 0, group));
  // 16-byte pieces of q, the cache and the output; the other kernels take what is not aligned.  Below four rows a row tile is
  // mostly empty: 2 rows x 4096 fp16 keys 35.7 us, chunk kernel 28.2.
  const double products = static_cast<double>(p.m) * span * p.heads * p.head_dim;
  if (kvkind == kKvF32 || p.m < 4 || products < tile_least(kvkind == kKvF16, p.m) || !aligned16(p.q) || !aligned16(p.k) ||
      !aligned16(p.v) || !aligned16(out))
    return kUnsupportedFeature;
  if (!writes_apart(kvkind, p, out, gate)) return kUnsupportedFeature;
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
