// Device and host helpers shared by the tcgen05 attention kernels (forward and backward translation units).
#pragma once
#include "attn_common.cuh"
#include "tc_common.cuh"
#include "tc_runtime.h"

namespace ptj {
namespace attn_tc {

using namespace tc;

constexpr int T = 128;                  // tile edge along queries and keys
constexpr int kSubBytes = T * 64 * 2;   // one [128][64] bf16 sub-tile: a [128][DHP] operand is DHP / 64 of them
constexpr int kPBytes = 2 * kSubBytes;  // one [128][128] bf16 tile of probabilities or score gradients
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

struct RowView {  // a [batch, heads, seq, d_head] view with d_head contiguous
  __nv_bfloat16* base;
  int64_t sb, sh, sr;
  __device__ __forceinline__ __nv_bfloat16* row(int64_t b, int64_t h, int64_t r) const {
    return base + b * sb + h * sh + r * sr;
  }
};

struct AttnParams {
  int S, H, BH, nq;  // nq = ceil(S / T): rows beyond S are zero-filled by the TMA copies and never stored
  int D;             // head size, a multiple of 8 up to DHP; columns beyond it are zero-filled as well
  float scale_log2;  // log2(e) / sqrt(d_head)
  float scale;       // 1 / sqrt(d_head)
  AttnDropout dr;
  const uint4* keep_bits;  // optional precomputed keep flags, one uint4 per (batch*head, tile, row): see attn_keep_bits_tc
  const int32_t* kstart;   // optional [batch, seq]: first key a query row may attend to (document start); NULL = 0
  unsigned int* fault;
};

// Philox round keys of a seed (round r uses rk[2r], rk[2r+1]): the same for every call of a kernel, so one thread
// writes them to shared memory at start-up, after resolving the seed argument (it may be the address of the seed).
__device__ __forceinline__ void philox_round_keys(uint64_t seed_arg, uint32_t* rk) {
  const uint64_t seed = resolve_seed(seed_arg);
  for (int r = 0; r < 10; ++r) {
    rk[2 * r] = static_cast<uint32_t>(seed) + static_cast<uint32_t>(r) * 0x9E3779B9u;
    rk[2 * r + 1] = static_cast<uint32_t>(seed >> 32) + static_cast<uint32_t>(r) * 0xBB67AE85u;
  }
}
// philox4x32_10 of common.cuh with the key schedule taken from a table
__device__ __forceinline__ void philox_rk(const uint32_t* rk, uint64_t ctr, uint32_t stream_id, uint32_t (&out)[4]) {
  uint32_t c0 = static_cast<uint32_t>(ctr), c1 = static_cast<uint32_t>(ctr >> 32), c2 = stream_id, c3 = 0x5054'4a31u;
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    const uint64_t p0 = static_cast<uint64_t>(0xD2511F53u) * c0;
    const uint64_t p1 = static_cast<uint64_t>(0xCD9E8D57u) * c2;
    const uint32_t n0 = static_cast<uint32_t>(p1 >> 32) ^ c1 ^ rk[2 * r];
    const uint32_t n2 = static_cast<uint32_t>(p0 >> 32) ^ c3 ^ rk[2 * r + 1];
    c1 = static_cast<uint32_t>(p1);
    c3 = static_cast<uint32_t>(p0);
    c0 = n0;
    c2 = n2;
  }
  out[0] = c0; out[1] = c1; out[2] = c2; out[3] = c3;
}

// Position of the 16-byte vector that holds columns [8 c8, 8 c8 + 8) of row r in a [128][128] bf16 tile stored as two
// [128][64] 128-byte-swizzled sub-tiles.
__device__ __forceinline__ uint8_t* p_vec(uint8_t* tile, int r, int c8) {
  return tile + (c8 >> 3) * kSubBytes + r * 128 + (((c8 & 7) ^ (r & 7)) << 4);
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<const uint32_t*>(&h);
}
__device__ __forceinline__ float bf16_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf16_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

// Eight floats -> the PARTS bf16 operands they are multiplied as, packed in pairs. One part: rounded to bf16. Three parts:
// the bf16 value nearest to x, the one nearest to what is left, and the one nearest to what is left then: 24 significant
// bits, those of a float32.
template <int PARTS>
__device__ __forceinline__ void split8(const float* v, uint32_t (&w)[PARTS][4]) {
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = v[2 * i], b = v[2 * i + 1];
#pragma unroll
    for (int p = 0; p < PARTS; ++p) {
      w[p][i] = pack_bf16(a, b);
      if (p + 1 < PARTS) {
        a -= bf16_lo(w[p][i]);
        b -= bf16_hi(w[p][i]);
      }
    }
  }
}
template <int PARTS>
__device__ __forceinline__ void store8(uint8_t* tile, int r, int c8, const uint32_t (&w)[PARTS][4]) {
#pragma unroll
  for (int p = 0; p < PARTS; ++p)
    *reinterpret_cast<uint4*>(p_vec(tile + p * kPBytes, r, c8)) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// Byte k of (x, y) with its sign bit copied to every bit, for each nibble 8 | k of the selector.
__device__ __forceinline__ uint32_t prmt_sign(uint32_t x, uint32_t y, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(x), "r"(y), "r"(sel));
  return r;
}
// Masks from a word of flags, i a compile-time constant: all ones where the flag is set. A permutation that replicates
// sign bits makes one from the word shifted so that the flag is the sign of its byte; the eight shifts are shared.
// Flags 2 i and 2 i + 1 in the halves of a word (for packed bf16) ...
__device__ __forceinline__ uint32_t pair_mask(uint32_t flags, int i) {
  const uint32_t k = static_cast<uint32_t>(i) >> 2;
  return prmt_sign(flags << (7 - 2 * (i & 3)), flags << (6 - 2 * (i & 3)), 0xcc88u + k * 0x1111u);
}
// ... and flag i in a whole word (for a float).
__device__ __forceinline__ float masked(float x, uint32_t flags, int i) {
  const uint32_t y = flags << (7 - (i & 7));
  return __uint_as_float(__float_as_uint(x) & prmt_sign(y, y, 0x8888u + (static_cast<uint32_t>(i) >> 3) * 0x1111u));
}

// bit i set: element i (0 <= i < 32) lies in [first, last], both relative to the same origin
__device__ __forceinline__ uint32_t range_bits(int first, int last) {
  const int n = min(max(last + 1, 0), 32), m = min(max(first, 0), 32);
  const uint32_t below_n = n >= 32 ? 0xffffffffu : (1u << n) - 1u;
  const uint32_t below_m = m >= 32 ? 0xffffffffu : (1u << m) - 1u;
  return below_n & ~below_m;
}

// Replaces the elements of a 16-byte vector in shared memory that are infinite or NaN by zero; true if there was one. A
// masked probability is an exact zero, but zero times an infinity or a NaN is a NaN: operands of a sum over masked entries
// pass through here, and what such an element would have reached is put back afterwards.
__device__ __forceinline__ bool zero_nonfinite(uint8_t* vec) {
  const uint4 x = *reinterpret_cast<const uint4*>(vec);
  uint32_t w[4] = {x.x, x.y, x.z, x.w}, m = 0u;
#pragma unroll
  for (int i = 0; i < 4; ++i) m = __vmaxu2(m, w[i] & 0x7fff7fffu);
  if ((m & 0xffffu) < 0x7f80u && (m >> 16) < 0x7f80u) return false;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    if ((w[i] & 0x7f80u) == 0x7f80u) w[i] &= 0xffff0000u;
    if ((w[i] & 0x7f800000u) == 0x7f800000u) w[i] &= 0xffffu;
  }
  *reinterpret_cast<uint4*>(vec) = make_uint4(w[0], w[1], w[2], w[3]);
  return true;
}

// 2^x on the special-function unit (inputs here are <= 0 or small; subnormal results flush to zero)
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// NCALL consecutive counters at once, rounds in a rolled loop (small code, the calls give the instruction-level
// parallelism), round keys read from shared memory (rk_s[2r], rk_s[2r+1]).
template <int NCALL>
__device__ __forceinline__ void philox_rolled(const uint32_t* rk_s, uint64_t ctr0, uint32_t stream_id, uint32_t (&out)[NCALL][4]) {
  uint32_t c0[NCALL], c1[NCALL], c2[NCALL], c3[NCALL];
#pragma unroll
  for (int q = 0; q < NCALL; ++q) {
    const uint64_t ctr = ctr0 + q;
    c0[q] = static_cast<uint32_t>(ctr);
    c1[q] = static_cast<uint32_t>(ctr >> 32);
    c2[q] = stream_id;
    c3[q] = 0x5054'4a31u;
  }
#pragma unroll 1
  for (int r = 0; r < 10; ++r) {
    const uint32_t k0 = rk_s[2 * r], k1 = rk_s[2 * r + 1];
#pragma unroll
    for (int q = 0; q < NCALL; ++q) {
      const uint64_t p0 = static_cast<uint64_t>(0xD2511F53u) * c0[q];
      const uint64_t p1 = static_cast<uint64_t>(0xCD9E8D57u) * c2[q];
      const uint32_t n0 = static_cast<uint32_t>(p1 >> 32) ^ c1[q] ^ k0;
      const uint32_t n2 = static_cast<uint32_t>(p0 >> 32) ^ c3[q] ^ k1;
      c1[q] = static_cast<uint32_t>(p1);
      c3[q] = static_cast<uint32_t>(p0);
      c0[q] = n0;
      c2[q] = n2;
    }
  }
#pragma unroll
  for (int q = 0; q < NCALL; ++q) {
    out[q][0] = c0[q]; out[q][1] = c1[q]; out[q][2] = c2[q]; out[q][3] = c3[q];
  }
}

// flags of the eight 16-bit lanes of one call (low half of word e / 2 for even e, high half for odd): set when >= threshold
__device__ __forceinline__ uint32_t keep_flags8(const uint32_t (&w)[4], uint32_t thr_hi) {
  uint32_t bits = 0u;
#pragma unroll
  for (int e = 0; e < 4; ++e) {
    bits |= ((w[e] << 16) >= thr_hi ? 1u : 0u) << (2 * e);
    bits |= (w[e] >= thr_hi ? 1u : 0u) << (2 * e + 1);
  }
  return bits;
}
// Keep flags of 32 consecutive elements from flat index idx0 on. A call yields the flags of eight elements from a multiple
// of eight on; where idx0 is none (rows of a sequence that is no multiple of eight) a fifth call fills the word.
__device__ __forceinline__ uint32_t keep_word(const uint32_t* rk_s, uint64_t idx0, uint32_t stream_id, uint32_t thr_hi) {
  uint32_t r[4][4], word = 0u;
  philox_rolled<4>(rk_s, idx0 >> 3, stream_id, r);
#pragma unroll
  for (int q = 0; q < 4; ++q) word |= keep_flags8(r[q], thr_hi) << (8 * q);
  const uint32_t shift = static_cast<uint32_t>(idx0) & 7u;
  if (shift != 0u) {
    uint32_t t[1][4];
    philox_rolled<1>(rk_s, (idx0 >> 3) + 4, stream_id, t);
    word = __funnelshift_r(word, keep_flags8(t[0], thr_hi), shift);
  }
  return word;
}

// packed pairs of floats for the two-wide fp32 instructions of sm_100 (fma.rn.f32x2, add.f32x2)
__device__ __forceinline__ uint64_t pack2(float lo, float hi) {
  uint64_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ void unpack2(uint64_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
  uint64_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ float max3(float a, float b, float c) {
  float r;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
  return r;
}

// descriptors of the operand flavours used below (all tiles are 128-byte swizzled, 8-line groups 1024 B apart)
__device__ __forceinline__ uint64_t desc_kmajor(uint32_t tile, int k16) {  // [128 rows][64-wide sub-tiles], K = columns
  return smem_desc_sw128(tile + (k16 >> 2) * kSubBytes + (k16 & 3) * 32, 16, 1024);
}
__device__ __forceinline__ uint64_t desc_rows_as_k(uint32_t tile, int k16) {  // the same bytes, K = rows, MN = columns
  return smem_desc_sw128(tile + k16 * 2048, kSubBytes, 1024);
}

__device__ __forceinline__ uint8_t* align1024(uint8_t* raw) {
  return raw + ((1024u - (smem_u32(raw) & 1023u)) & 1023u);
}

// ---- host side -------------------------------------------------------------------------------------------------
inline bool make_map(CUtensorMap* m, const void* base, const ptj_attn_shape& sh, const int64_t (&st)[3]) {
  const uint64_t dims[4] = {static_cast<uint64_t>(sh.d_head), static_cast<uint64_t>(sh.seq),
                            static_cast<uint64_t>(sh.heads), static_cast<uint64_t>(sh.batch)};
  // a size-1 dimension may come with any stride; the encoder wants positive multiples of 16 bytes
  auto fix = [&](int64_t s, int64_t n) { return static_cast<uint64_t>(n > 1 ? s : T) * 2; };
  const uint64_t strides[3] = {fix(st[2], sh.seq), fix(st[1], sh.heads), fix(st[0], sh.batch)};
  const uint32_t box[4] = {64, T, 1, 1};
  return make_tmap_bf16(m, base, 4, dims, strides, box);
}
// one thread: [128][DHP] rows from `row` on of a head, as DHP / 64 sub-tiles
template <int DHP>
__device__ __forceinline__ void load_rows(uint8_t* dst, const CUtensorMap* m, uint64_t* bar, int row, int h, int b) {
#pragma unroll
  for (int x = 0; x < DHP / 64; ++x) tma_load_4d(dst + x * kSubBytes, m, bar, 64 * x, row, h, b);
}

inline RowView make_view(const void* base, const int64_t (&st)[3]) {
  return RowView{static_cast<__nv_bfloat16*>(const_cast<void*>(base)), st[0], st[1], st[2]};
}

inline AttnParams make_params(const ptj_attn_shape& sh, const AttnDropout& dr) {
  AttnParams p{};
  p.S = static_cast<int>(sh.seq);
  p.H = static_cast<int>(sh.heads);
  p.BH = static_cast<int>(sh.batch * sh.heads);
  p.nq = (p.S + T - 1) / T;
  p.D = static_cast<int>(sh.d_head);
  p.scale = 1.f / sqrtf(static_cast<float>(p.D));
  p.scale_log2 = p.scale * kLog2e;
  p.dr = dr;
  p.fault = tc::fault_word();
  return p;
}

}  // namespace attn_tc
}  // namespace ptj
