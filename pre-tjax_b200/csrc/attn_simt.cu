// Causal attention forward / backward in float32 arithmetic on CUDA cores, for any head size up to 128, any sequence
// length and any strides. Semantics: model_triton.py:510-517, 608-611 (forward), :550-577, 801-811 (backward); dropout
// acts on the probabilities and is not rescaled. No atomics: the backward is split into a dQ pass and a dK/dV pass that
// both recompute the probabilities from the saved row maximum and row sum.
//
// A thread block owns a tile of 64 query (dK/dV pass: key) rows and sweeps 64-row tiles of the other side through shared
// memory. 16 x (64 / kR) threads each form a kR x 4 block of the 64 x 64 scores, and a kR x (DP / 16) block of every
// output tile, in registers: two or three 16-byte shared loads per 32 multiply-adds. Score products pack neighbouring
// d into the two-wide FMA straight from those loads. Bound by the FP32 pipe (a warp per row with scalar global loads
// was bound by the load/store unit instead). Measured, float32, forward / backward: [8, 12, 512, 64] with dropout and
// document masks 88 / 265 us (36 / 43 TFLOP/s of the causal half), where a warp per row with a Philox call per probability
// took 2526 / 16152 us; [4, 12, 512, 64] without dropout 84 / 264 us, forward 1900 us before. kR = 4: twice the warps of
// kR = 8, which needs 255 registers and measured 98 / 314 and 90 / 294 us there, 23 / 75 us against 17 / 58 us at
// [2, 12, 128, 64]. The dK/dV kernel is held to two blocks per SM: left alone it took 234 registers and one block, 317 us
// at the first of these sizes.
#include "attn_common.cuh"

namespace ptj {
namespace {

constexpr int kMaxD = 128;
constexpr int kB = 64;         // tile edge along queries and keys
constexpr int kPS = kB + 4;    // row stride of a [64][64] tile in shared memory
constexpr int kR = 4;          // rows of a tile per thread
constexpr int kFlagStride = 12;  // bytes per row of keep flags: 64 flags that may start anywhere in a byte

template <int DP>
struct Tile {
  static constexpr int kThreads = 16 * kB / kR;
  static constexpr int kLd = DP + 4;             // row stride (words): 16-byte reads of 8 consecutive rows hit 32 banks
  static constexpr int kWords = kB * kLd;
  static constexpr int kCols = DP / 16;          // output columns of a thread
  static constexpr int kVec = kCols < 4 ? kCols : 4;
  static __device__ __forceinline__ int col(int c, int tx) { return (c / kVec) * (16 * kVec) + tx * kVec + c % kVec; }
};

// four consecutive elements of a row (zeros from element n on); vec: 4 elements are one aligned vector
template <typename T>
__device__ __forceinline__ float4 load4(const T* p, int n, bool vec) {
  float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
  if (vec) {
    if (n >= 4) {
      if constexpr (sizeof(T) == 4) {
        v = *reinterpret_cast<const float4*>(p);
      } else {
        const uint2 t = *reinterpret_cast<const uint2*>(p);
        v = make_float4(__uint_as_float(t.x << 16), __uint_as_float(t.x & 0xffff0000u), __uint_as_float(t.y << 16),
                        __uint_as_float(t.y & 0xffff0000u));
      }
    }
  } else {
    if (n > 0) v.x = Elem<T>::load(p);
    if (n > 1) v.y = Elem<T>::load(p + 1);
    if (n > 2) v.z = Elem<T>::load(p + 2);
    if (n > 3) v.w = Elem<T>::load(p + 3);
  }
  return v;
}

// A masked probability is an exact zero, but zero times an infinity or a NaN is a NaN: a tile that holds one is multiplied
// with the masked entries left out (mul_*_masked), so that a row reads only what it attends. The loads form this sum of
// zeros on the side; it is a NaN where an element is not finite. Cost: 262 -> 265 us in the backward kernels at
// [8, 12, 512, 64], none in the forward kernel.
__device__ __forceinline__ float zero_sum(float z, const float4& v) {
  return fmaf(v.x, 0.f, fmaf(v.y, 0.f, fmaf(v.z, 0.f, fmaf(v.w, 0.f, z))));
}

// rows [r0, r0 + 64) of a [seq][D] view, zero-filled to [64][DP]; true when this thread met an element that is not finite
template <typename T, int DP>
__device__ __forceinline__ bool load_tile(float* dst, const T* base, int64_t rs, int64_t r0, int64_t S, int D, bool vec) {
  constexpr int kC4 = DP / 4;
  float z = 0.f;
#pragma unroll 4
  for (int idx = threadIdx.x; idx < kB * kC4; idx += Tile<DP>::kThreads) {
    const int row = idx / kC4, c = idx % kC4 * 4;
    const int n = r0 + row < S ? D - c : 0;
    const float4 v = load4(base + (r0 + row) * rs + c, n, vec);
    *reinterpret_cast<float4*>(dst + row * Tile<DP>::kLd + c) = v;
    z = zero_sum(z, v);
  }
  return z != 0.f;  // (a NaN is unequal to everything)
}

// the same for dO, with delta[row] = sum_d dO O on the side
template <typename T, int DP>
__device__ __forceinline__ bool load_tile_delta(float* dst, float* delta, const T* g, const T* o, int64_t rs, int64_t r0,
                                                int64_t S, int D, bool vec) {
  constexpr int kC4 = DP / 4;  // 8, 16 or 32 consecutive lanes hold a row
  float z = 0.f;
#pragma unroll 4
  for (int idx = threadIdx.x; idx < kB * kC4; idx += Tile<DP>::kThreads) {
    const int row = idx / kC4, c = idx % kC4 * 4;
    const int n = r0 + row < S ? D - c : 0;
    const float4 a = load4(g + (r0 + row) * rs + c, n, vec), b = load4(o + (r0 + row) * rs + c, n, vec);
    *reinterpret_cast<float4*>(dst + row * Tile<DP>::kLd + c) = a;
    z = zero_sum(z, a);
    float s = fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w)));
#pragma unroll
    for (int off = kC4 / 2; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
    if (idx % kC4 == 0) delta[row] = s;
  }
  return z != 0.f;
}

// keep flags of the 64 x 64 tile at (r0, j0): nine bytes per row from the Philox call that holds the row's first element
__device__ __forceinline__ void draw_flags(uint8_t* flags, const AttnDropout& dr, int64_t bh, int64_t S, int64_t r0,
                                           int64_t j0, int nthreads) {
  for (int x = threadIdx.x; x < kB * 9; x += nthreads) {
    const int row = x / 9, call = x % 9;
    const uint64_t idx0 = (static_cast<uint64_t>(bh) * S + r0 + row) * S + j0;
    flags[row * kFlagStride + call] =
        static_cast<uint8_t>(dropout_keep_bits8(dr.seed, dr.stream_id, (idx0 >> 3) + call, dr.thr16));
  }
}
__device__ __forceinline__ bool flag_at(const uint8_t* row_flags, int bit) { return (row_flags[bit >> 3] >> (bit & 7)) & 1; }

// acc[r][c] = sum_d a[ty * kR + r][d] * b[tx + 16 c][d]
template <int DP>
__device__ __forceinline__ void mul_nt(float (&out)[kR][4], const float* a, const float* b, int tx, int ty) {
  constexpr int ld = Tile<DP>::kLd;
  uint64_t acc[kR][4];
#pragma unroll
  for (int r = 0; r < kR; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) acc[r][c] = 0ull;
#pragma unroll 2
  for (int d = 0; d < DP; d += 4) {
    ulonglong2 y[4];
#pragma unroll
    for (int c = 0; c < 4; ++c) y[c] = *reinterpret_cast<const ulonglong2*>(b + (tx + 16 * c) * ld + d);
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(a + (ty * kR + r) * ld + d);
#pragma unroll
      for (int c = 0; c < 4; ++c) acc[r][c] = f2_fma(x.y, y[c].y, f2_fma(x.x, y[c].x, acc[r][c]));
    }
  }
#pragma unroll
  for (int r = 0; r < kR; ++r)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      float lo, hi;
      f2_unpack(acc[r][c], lo, hi);
      out[r][c] = lo + hi;
    }
}

// one row of an output tile's operand: this thread's columns
template <int DP>
__device__ __forceinline__ void load_cols(float (&v)[Tile<DP>::kCols], const float* row, int tx) {
  using TT = Tile<DP>;
#pragma unroll
  for (int c = 0; c < TT::kCols; c += TT::kVec) {
    if constexpr (TT::kVec == 4) {
      const float4 t = *reinterpret_cast<const float4*>(row + TT::col(c, tx));
      v[c] = t.x; v[c + 1] = t.y; v[c + 2] = t.z; v[c + 3] = t.w;
    } else {
      const float2 t = *reinterpret_cast<const float2*>(row + TT::col(c, tx));
      v[c] = t.x; v[c + 1] = t.y;
    }
  }
}

// acc[r][.] += sum_k w[ty * kR + r][k] * x[k][cols]   (rows of w written by the same half-warp)
template <int DP>
__device__ __forceinline__ void mul_nn(float (&acc)[kR][Tile<DP>::kCols], const float* w, const float* x, int tx, int ty) {
  constexpr int kCols = Tile<DP>::kCols;
#pragma unroll 1
  for (int k = 0; k < kB; k += 4) {
    float4 p[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) p[r] = *reinterpret_cast<const float4*>(w + (ty * kR + r) * kPS + k);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk) {
      float v[kCols];
      load_cols<DP>(v, x + (k + kk) * Tile<DP>::kLd, tx);
#pragma unroll
      for (int r = 0; r < kR; ++r) {
        const float pr = kk == 0 ? p[r].x : (kk == 1 ? p[r].y : (kk == 2 ? p[r].z : p[r].w));
#pragma unroll
        for (int c = 0; c < kCols; ++c) acc[r][c] = fmaf(pr, v[c], acc[r][c]);
      }
    }
  }
}

// acc[r][.] += sum_q w[q][ty * kR + r] * x[q][cols]
template <int DP>
__device__ __forceinline__ void mul_tn(float (&acc)[kR][Tile<DP>::kCols], const float* w, const float* x, int tx, int ty) {
  constexpr int kCols = Tile<DP>::kCols;
#pragma unroll 2
  for (int q = 0; q < kB; ++q) {
    float p[kR], v[kCols];
#pragma unroll
    for (int r = 0; r < kR; r += 4) {
      const float4 t = *reinterpret_cast<const float4*>(w + q * kPS + ty * kR + r);
      p[r] = t.x; p[r + 1] = t.y; p[r + 2] = t.z; p[r + 3] = t.w;
    }
    load_cols<DP>(v, x + q * Tile<DP>::kLd, tx);
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
      for (int c = 0; c < kCols; ++c) acc[r][c] = fmaf(p[r], v[c], acc[r][c]);
  }
}

// The two sums over unmasked entries alone, on(r, k) and on(q, r): for tiles with elements that are not finite.
template <int DP, typename On>
__device__ __forceinline__ void mul_nn_masked(float (&acc)[kR][Tile<DP>::kCols], const float* w, const float* x, int tx, int ty,
                                              On&& on) {
  constexpr int kCols = Tile<DP>::kCols;
#pragma unroll 1
  for (int k = 0; k < kB; ++k) {
    float v[kCols];
    load_cols<DP>(v, x + k * Tile<DP>::kLd, tx);
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      if (!on(r, k)) continue;
      const float p = w[(ty * kR + r) * kPS + k];
#pragma unroll
      for (int c = 0; c < kCols; ++c) acc[r][c] = fmaf(p, v[c], acc[r][c]);
    }
  }
}
template <int DP, typename On>
__device__ __forceinline__ void mul_tn_masked(float (&acc)[kR][Tile<DP>::kCols], const float* w, const float* x, int tx, int ty,
                                              On&& on) {
  constexpr int kCols = Tile<DP>::kCols;
#pragma unroll 1
  for (int q = 0; q < kB; ++q) {
    float v[kCols];
    load_cols<DP>(v, x + q * Tile<DP>::kLd, tx);
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      if (!on(q, r)) continue;
      const float p = w[q * kPS + ty * kR + r];
#pragma unroll
      for (int c = 0; c < kCols; ++c) acc[r][c] = fmaf(p, v[c], acc[r][c]);
    }
  }
}

// this thread's block of an output tile; mul[r] scales a row. patch: only elements that are not finite, here or in memory
template <typename T, int DP>
__device__ __forceinline__ void store_rows(T* base, int64_t rs, int64_t r0, int64_t S, int D, bool vec,
                                           const float (&acc)[kR][Tile<DP>::kCols], const float (&mul)[kR], int tx, int ty,
                                           bool patch = false) {
  using TT = Tile<DP>;
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int64_t i = r0 + ty * kR + r;
    if (i >= S) continue;
    T* row = base + i * rs;
#pragma unroll
    for (int c = 0; c < TT::kCols; c += TT::kVec) {
      const int col = TT::col(c, tx);
      if (patch) {
        for (int e = 0; e < TT::kVec; ++e) {
          const float x = acc[r][c + e] * mul[r];
          if (col + e < D && !(isfinite(x) && isfinite(Elem<T>::load(row + col + e)))) Elem<T>::store(row + col + e, x);
        }
      } else if (sizeof(T) == 4 && TT::kVec == 4 && vec) {
        if (col < D)
          *reinterpret_cast<float4*>(row + col) =
              make_float4(acc[r][c] * mul[r], acc[r][c + 1] * mul[r], acc[r][c + 2 < TT::kCols ? c + 2 : c] * mul[r],
                          acc[r][c + 3 < TT::kCols ? c + 3 : c] * mul[r]);
      } else {
#pragma unroll
        for (int e = 0; e < TT::kVec; ++e)
          if (col + e < D) Elem<T>::store(row + col + e, acc[r][c + e] * mul[r]);
      }
    }
  }
}

__device__ __forceinline__ float half_warp_max(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float half_warp_sum(float v) {
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

template <typename T>
struct FwdArgs {
  const T *q, *k, *v;
  T* o;
  float *row_max, *row_sum;
  const int32_t* kstart;
  ptj_attn_shape sh;
  float scale;
  int nq;
  bool vec;
  AttnDropout dr;
};

// Block = one query tile of one (batch, head), the longest rows first. Online softmax over the key tiles.
template <typename T, int DP>
__global__ void __launch_bounds__(Tile<DP>::kThreads)
attn_fwd_simt_kernel(const FwdArgs<T> a) {
  grid_dep_sync();
  using TT = Tile<DP>;
  extern __shared__ __align__(16) float smem[];
  float* q_s = smem;
  float* v_s = q_s + TT::kWords;
  float* k_s = v_s + TT::kWords;
  // the probabilities take the place of the key tile (for 32-wide heads a [64][68] tile is the larger of the two)
  float* p_s = k_s;
  uint8_t* flags = reinterpret_cast<uint8_t*>(k_s + (TT::kWords > kB * kPS ? TT::kWords : kB * kPS));
  __shared__ int first_key;
  AttnDropout dr = a.dr;
  const bool drop = dr.train && dr.thr16 != 0u;
  if (drop) dr.seed = resolve_seed(dr.seed);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t S = a.sh.seq;
  const int D = static_cast<int>(a.sh.d_head);
  const int64_t nbh = a.sh.batch * a.sh.heads;
  const int qt = a.nq - 1 - static_cast<int>(blockIdx.x / nbh);
  const int64_t bh = blockIdx.x % nbh, b = bh / a.sh.heads, h = bh % a.sh.heads;
  const int64_t r0 = static_cast<int64_t>(qt) * kB;
  const T* kb = a.k + b * a.sh.k_strides[0] + h * a.sh.k_strides[1];
  const T* vb = a.v + b * a.sh.v_strides[0] + h * a.sh.v_strides[1];
  load_tile<T, DP>(q_s, a.q + b * a.sh.q_strides[0] + h * a.sh.q_strides[1], a.sh.q_strides[2], r0, S, D, a.vec);

  // row i attends keys [ks, i]; ks > i (padding, rows beyond the sequence): nothing
  int64_t ks[kR];
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int64_t i = r0 + ty * kR + r;
    ks[r] = i >= S ? i + 1 : (a.kstart != nullptr ? a.kstart[b * S + i] : 0);
  }
  int kt0 = 0;
  if (a.kstart != nullptr) {  // key tiles before every row's first key are skipped
    if (threadIdx.x == 0) first_key = 0x7fffffff;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kR; ++r)
      if (tx == 0 && ks[r] <= r0 + ty * kR + r) atomicMin(&first_key, static_cast<int>(ks[r] > 0 ? ks[r] : 0));
    __syncthreads();
    kt0 = first_key / kB;
  }

  float m[kR], l[kR], acc[kR][TT::kCols];
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    m[r] = -INFINITY;
    l[r] = 0.f;
#pragma unroll
    for (int c = 0; c < TT::kCols; ++c) acc[r][c] = 0.f;
  }
  for (int kt = kt0; kt <= qt; ++kt) {
    const int64_t j0 = static_cast<int64_t>(kt) * kB;
    __syncthreads();
    load_tile<T, DP>(k_s, kb, a.sh.k_strides[2], j0, S, D, a.vec);
    const bool odd_v = load_tile<T, DP>(v_s, vb, a.sh.v_strides[2], j0, S, D, a.vec);
    if (drop) draw_flags(flags, dr, bh, S, r0, j0, TT::kThreads);
    const bool masked = __syncthreads_or(odd_v);
    float s[kR][4];
    mul_nt<DP>(s, q_s, k_s, tx, ty);
    __syncthreads();  // the key tile is free
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int64_t i = r0 + ty * kR + r;
      float mx = -INFINITY;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int64_t j = j0 + tx + 16 * c;
        s[r][c] = (j <= i && j >= ks[r]) ? s[r][c] * a.scale : -INFINITY;
        mx = fmaxf(mx, s[r][c]);
      }
      const float mnew = fmaxf(m[r], half_warp_max(mx));
      const float ref = mnew == -INFINITY ? 0.f : mnew;  // a row that has met none of its keys yet
      const float corr = expf(m[r] - ref);
      float sum = 0.f;
      const int shift = static_cast<int>(((static_cast<uint64_t>(bh) * S + i) * S + j0) & 7u);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        float p = expf(s[r][c] - ref);
        sum += p;
        if (drop) {
          if (!flag_at(flags + (ty * kR + r) * kFlagStride, tx + 16 * c + shift)) p = 0.f;
        } else if (!dr.train) {
          p *= dr.eval_scale;
        }
        p_s[(ty * kR + r) * kPS + tx + 16 * c] = p;
      }
      l[r] = l[r] * corr + half_warp_sum(sum);
#pragma unroll
      for (int c = 0; c < TT::kCols; ++c) acc[r][c] *= corr;
      m[r] = mnew;
    }
    __syncwarp();  // a row's probabilities are written and read by the same half-warp
    if (!masked) mul_nn<DP>(acc, p_s, v_s, tx, ty);
    else mul_nn_masked<DP>(acc, p_s, v_s, tx, ty, [&](int r, int k) { return j0 + k <= r0 + ty * kR + r && j0 + k >= ks[r]; });
  }
  float inv[kR];
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int64_t i = r0 + ty * kR + r;
    const bool empty = ks[r] > i;  // zero output, neutral statistics
    inv[r] = empty ? 0.f : 1.f / l[r];
    if (empty) {
#pragma unroll
      for (int c = 0; c < TT::kCols; ++c) acc[r][c] = 0.f;
    }
    if (tx == 0 && i < S) {
      a.row_max[bh * S + i] = empty ? 0.f : m[r];
      a.row_sum[bh * S + i] = empty ? 1.f : l[r];
    }
  }
  store_rows<T, DP>(a.o + b * a.sh.o_strides[0] + h * a.sh.o_strides[1], a.sh.o_strides[2], r0, S, D, a.vec, acc, inv,
                       tx, ty);
}

template <typename T>
struct BwdArgs {
  const T *d_o, *q, *k, *v, *o;
  const float *row_max, *row_sum;
  T *dq, *dk, *dv;
  const int32_t* kstart;
  const unsigned int* patch;  // optional: the results are there; when this word is set, put in what is not finite
  ptj_attn_shape sh, dsh;
  float scale;
  int nq;
  bool vec;
  AttnDropout dr;
};

// per-row constants of a query tile in shared memory
struct RowConst {
  float delta[kB], m[kB], inv_l[kB];
  int ks[kB];  // first key relative to the sequence; beyond the row's own position: the row attends nothing
};
template <typename T>
__device__ __forceinline__ void load_row_const(RowConst& rc, const BwdArgs<T>& a, int64_t b, int64_t bh, int64_t r0) {
  if (threadIdx.x < kB) {
    const int64_t i = r0 + threadIdx.x, S = a.sh.seq;
    const bool real = i < S;
    rc.m[threadIdx.x] = real ? a.row_max[bh * S + i] : 0.f;
    rc.inv_l[threadIdx.x] = real ? 1.f / a.row_sum[bh * S + i] : 0.f;
    rc.ks[threadIdx.x] = !real ? 0x7fffffff : (a.kstart != nullptr ? a.kstart[b * S + i] : 0);
  }
}

// Probabilities and score gradients of this thread's kR x 4 block: s holds Q K^T on entry and dropout(P) on exit, dp holds
// dO V^T on entry and dS = P o (dP o keep - delta) * scale on exit.
template <typename T>
__device__ __forceinline__ void p_and_ds(float (&s)[kR][4], float (&dp)[kR][4], const RowConst& rc, const uint8_t* flags,
                                         bool drop, const BwdArgs<T>& a, int64_t bh, int64_t r0, int64_t j0, int tx, int ty) {
  const int64_t S = a.sh.seq;
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    const int row = ty * kR + r;
    const int64_t i = r0 + row;
    const float m = rc.m[row], inv_l = rc.inv_l[row], delta = rc.delta[row];
    const int64_t ks = rc.ks[row];
    const int shift = static_cast<int>(((static_cast<uint64_t>(bh) * S + i) * S + j0) & 7u);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const int64_t j = j0 + tx + 16 * c;
      const bool on = j <= i && j >= ks;
      const float p = on ? expf(s[r][c] * a.scale - m) * inv_l : 0.f;
      const float f = drop ? (flag_at(flags + row * kFlagStride, tx + 16 * c + shift) ? 1.f : 0.f)
                           : (a.dr.train ? 1.f : a.dr.eval_scale);
      dp[r][c] = on ? p * (dp[r][c] * f - delta) * a.scale : 0.f;
      s[r][c] = p * f;
    }
  }
}

// dQ: block = one query tile, the longest rows first; sweeps the key tiles.
template <typename T, int DP>
__global__ void __launch_bounds__(Tile<DP>::kThreads)
attn_dq_simt_kernel(const BwdArgs<T> a) {
  grid_dep_sync();
  if (a.patch != nullptr && *a.patch == 0u) return;
  using TT = Tile<DP>;
  extern __shared__ __align__(16) float smem[];
  float* q_s = smem;
  float* g_s = q_s + TT::kWords;
  float* k_s = g_s + TT::kWords;
  float* v_s = k_s + TT::kWords;
  float* ds_s = v_s + TT::kWords;
  uint8_t* flags = reinterpret_cast<uint8_t*>(ds_s + kB * kPS);
  __shared__ RowConst rc;
  __shared__ int first_key;
  AttnDropout dr = a.dr;
  const bool drop = dr.train && dr.thr16 != 0u;
  if (drop) dr.seed = resolve_seed(dr.seed);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t S = a.sh.seq;
  const int D = static_cast<int>(a.sh.d_head);
  const int64_t nbh = a.sh.batch * a.sh.heads;
  const int qt = a.nq - 1 - static_cast<int>(blockIdx.x / nbh);
  const int64_t bh = blockIdx.x % nbh, b = bh / a.sh.heads, h = bh % a.sh.heads;
  const int64_t r0 = static_cast<int64_t>(qt) * kB, o_off = b * a.sh.o_strides[0] + h * a.sh.o_strides[1];
  if (threadIdx.x == 0) first_key = 0x7fffffff;
  load_row_const(rc, a, b, bh, r0);
  load_tile<T, DP>(q_s, a.q + b * a.sh.q_strides[0] + h * a.sh.q_strides[1], a.sh.q_strides[2], r0, S, D, a.vec);
  load_tile_delta<T, DP>(g_s, rc.delta, a.d_o + o_off, a.o + o_off, a.sh.o_strides[2], r0, S, D, a.vec);
  __syncthreads();
  int kt0 = 0;
  if (a.kstart != nullptr) {
    if (threadIdx.x < kB && rc.ks[threadIdx.x] <= r0 + threadIdx.x)
      atomicMin(&first_key, rc.ks[threadIdx.x] > 0 ? rc.ks[threadIdx.x] : 0);
    __syncthreads();
    kt0 = first_key / kB;
  }
  float acc[kR][TT::kCols], one[kR];
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    one[r] = 1.f;
#pragma unroll
    for (int c = 0; c < TT::kCols; ++c) acc[r][c] = 0.f;
  }
  for (int kt = kt0; kt <= qt; ++kt) {
    const int64_t j0 = static_cast<int64_t>(kt) * kB;
    __syncthreads();
    const bool odd_k =
        load_tile<T, DP>(k_s, a.k + b * a.sh.k_strides[0] + h * a.sh.k_strides[1], a.sh.k_strides[2], j0, S, D, a.vec);
    load_tile<T, DP>(v_s, a.v + b * a.sh.v_strides[0] + h * a.sh.v_strides[1], a.sh.v_strides[2], j0, S, D, a.vec);
    if (drop) draw_flags(flags, dr, bh, S, r0, j0, TT::kThreads);
    const bool masked = __syncthreads_or(odd_k);
    float s[kR][4], dp[kR][4];
    mul_nt<DP>(s, q_s, k_s, tx, ty);
    mul_nt<DP>(dp, g_s, v_s, tx, ty);
    p_and_ds<T>(s, dp, rc, flags, drop, a, bh, r0, j0, tx, ty);
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) ds_s[(ty * kR + r) * kPS + tx + 16 * c] = dp[r][c];
    __syncwarp();  // a row is written and read by the same half-warp
    if (!masked) mul_nn<DP>(acc, ds_s, k_s, tx, ty);
    else mul_nn_masked<DP>(acc, ds_s, k_s, tx, ty, [&](int r, int k) {
      return j0 + k <= r0 + ty * kR + r && j0 + k >= rc.ks[ty * kR + r];
    });
    __syncwarp();
  }
  store_rows<T, DP>(a.dq + b * a.dsh.q_strides[0] + h * a.dsh.q_strides[1], a.dsh.q_strides[2], r0, S, D, a.vec, acc,
                       one, tx, ty, a.patch != nullptr);
}

// dK and dV: block = one key tile, the ones with the most query tiles first; sweeps the query tiles.
template <typename T, int DP>
__global__ void __launch_bounds__(Tile<DP>::kThreads, DP <= 64 ? 2 : 1)  // (wide heads: shared memory takes one block)
attn_dkv_simt_kernel(const BwdArgs<T> a) {
  grid_dep_sync();
  if (a.patch != nullptr && *a.patch == 0u) return;
  using TT = Tile<DP>;
  extern __shared__ __align__(16) float smem[];
  float* q_s = smem;
  float* g_s = q_s + TT::kWords;
  float* k_s = g_s + TT::kWords;
  float* v_s = k_s + TT::kWords;
  float* p_s = v_s + TT::kWords;
  float* ds_s = p_s + kB * kPS;
  uint8_t* flags = reinterpret_cast<uint8_t*>(ds_s + kB * kPS);
  __shared__ RowConst rc;
  AttnDropout dr = a.dr;
  const bool drop = dr.train && dr.thr16 != 0u;
  if (drop) dr.seed = resolve_seed(dr.seed);
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int64_t S = a.sh.seq;
  const int D = static_cast<int>(a.sh.d_head);
  const int64_t nbh = a.sh.batch * a.sh.heads;
  const int kt = static_cast<int>(blockIdx.x / nbh);
  const int64_t bh = blockIdx.x % nbh, b = bh / a.sh.heads, h = bh % a.sh.heads;
  const int64_t j0 = static_cast<int64_t>(kt) * kB, o_off = b * a.sh.o_strides[0] + h * a.sh.o_strides[1];
  load_tile<T, DP>(k_s, a.k + b * a.sh.k_strides[0] + h * a.sh.k_strides[1], a.sh.k_strides[2], j0, S, D, a.vec);
  load_tile<T, DP>(v_s, a.v + b * a.sh.v_strides[0] + h * a.sh.v_strides[1], a.sh.v_strides[2], j0, S, D, a.vec);
  float dk[kR][TT::kCols], dv[kR][TT::kCols], one[kR];
#pragma unroll
  for (int r = 0; r < kR; ++r) {
    one[r] = 1.f;
#pragma unroll
    for (int c = 0; c < TT::kCols; ++c) dk[r][c] = dv[r][c] = 0.f;
  }
  for (int qt = kt; qt < a.nq; ++qt) {
    const int64_t r0 = static_cast<int64_t>(qt) * kB;
    __syncthreads();
    load_row_const(rc, a, b, bh, r0);
    if (a.kstart != nullptr) {  // none of the tile's rows reaches into this key tile
      const bool reach = threadIdx.x < kB && rc.ks[threadIdx.x] <= r0 + threadIdx.x && rc.ks[threadIdx.x] < j0 + kB;
      if (!__syncthreads_or(reach)) continue;
    }
    const bool odd_q =
        load_tile<T, DP>(q_s, a.q + b * a.sh.q_strides[0] + h * a.sh.q_strides[1], a.sh.q_strides[2], r0, S, D, a.vec);
    const bool odd_g =
        load_tile_delta<T, DP>(g_s, rc.delta, a.d_o + o_off, a.o + o_off, a.sh.o_strides[2], r0, S, D, a.vec);
    if (drop) draw_flags(flags, dr, bh, S, r0, j0, TT::kThreads);
    const bool masked = __syncthreads_or(odd_q || odd_g);
    float s[kR][4], dp[kR][4];
    mul_nt<DP>(s, q_s, k_s, tx, ty);
    mul_nt<DP>(dp, g_s, v_s, tx, ty);
    p_and_ds<T>(s, dp, rc, flags, drop, a, bh, r0, j0, tx, ty);
#pragma unroll
    for (int r = 0; r < kR; ++r)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        p_s[(ty * kR + r) * kPS + tx + 16 * c] = s[r][c];
        ds_s[(ty * kR + r) * kPS + tx + 16 * c] = dp[r][c];
      }
    __syncthreads();
    if (!masked) {
      mul_tn<DP>(dv, p_s, g_s, tx, ty);
      mul_tn<DP>(dk, ds_s, q_s, tx, ty);
    } else {
      const auto on = [&](int q, int r) { return j0 + ty * kR + r <= r0 + q && j0 + ty * kR + r >= rc.ks[q]; };
      mul_tn_masked<DP>(dv, p_s, g_s, tx, ty, on);
      mul_tn_masked<DP>(dk, ds_s, q_s, tx, ty, on);
    }
  }
  store_rows<T, DP>(a.dv + b * a.dsh.v_strides[0] + h * a.dsh.v_strides[1], a.dsh.v_strides[2], j0, S, D, a.vec, dv,
                       one, tx, ty, a.patch != nullptr);
  store_rows<T, DP>(a.dk + b * a.dsh.k_strides[0] + h * a.dsh.k_strides[1], a.dsh.k_strides[2], j0, S, D, a.vec, dk,
                       one, tx, ty, a.patch != nullptr);
}

// every row starts on a multiple of four elements: rows are read as vectors
template <typename T>
bool rows_vectorise(const ptj_attn_shape& sh, const void* const* ptrs, int n) {
  if (sh.d_head % 4 != 0) return false;
  for (int i = 0; i < n; ++i)
    if (reinterpret_cast<uintptr_t>(ptrs[i]) % (4 * sizeof(T)) != 0) return false;
  for (int i = 0; i < 3; ++i)
    if (sh.q_strides[i] % 4 != 0 || sh.k_strides[i] % 4 != 0 || sh.v_strides[i] % 4 != 0 || sh.o_strides[i] % 4 != 0)
      return false;
  return true;
}

template <typename Args>
int launch_tiles(void (*kern)(const Args), int threads, size_t smem, const Args& a, cudaStream_t st) {
  const int64_t blocks = a.sh.batch * a.sh.heads * a.nq;
  if (blocks > 0x7fffffff) return PTJ_ERR_UNSUPPORTED;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)) != cudaSuccess) {
    (void)cudaGetLastError();
    return PTJ_ERR_LAUNCH;
  }
  launch_k(kern, static_cast<unsigned>(blocks), threads, smem, st, a);
  PTJ_CHECK_LAUNCH();
  return PTJ_OK;
}

constexpr size_t kFlagBytes = kB * kFlagStride;

template <typename T, int DP>
int run_fwd(const FwdArgs<T>& a, cudaStream_t st) {
  using TT = Tile<DP>;
  const size_t k_words = TT::kWords > kB * kPS ? TT::kWords : kB * kPS;
  return launch_tiles(attn_fwd_simt_kernel<T, DP>, TT::kThreads, (2 * TT::kWords + k_words) * 4 + kFlagBytes, a, st);
}

template <typename T, int DP>
int run_bwd(const BwdArgs<T>& a, cudaStream_t st) {
  using TT = Tile<DP>;
  const size_t tiles = 4 * TT::kWords * 4 + kFlagBytes, p = kB * kPS * 4;
  const int rc = launch_tiles(attn_dq_simt_kernel<T, DP>, TT::kThreads, tiles + p, a, st);
  if (rc != PTJ_OK) return rc;
  return launch_tiles(attn_dkv_simt_kernel<T, DP>, TT::kThreads, tiles + 2 * p, a, st);
}

template <typename T>
int fwd_typed(const void* q, const void* k, const void* v, void* o, float* row_max, float* row_sum,
              const int32_t* row_kstart, const ptj_attn_shape& sh, const AttnDropout& dr, cudaStream_t st) {
  const void* ptrs[4] = {q, k, v, o};
  const FwdArgs<T> a{static_cast<const T*>(q), static_cast<const T*>(k), static_cast<const T*>(v), static_cast<T*>(o),
                     row_max, row_sum, row_kstart, sh, 1.f / sqrtf(static_cast<float>(sh.d_head)),
                     static_cast<int>(ceil_div(sh.seq, kB)), rows_vectorise<T>(sh, ptrs, 4), dr};
  if (sh.d_head <= 32) return run_fwd<T, 32>(a, st);
  if (sh.d_head <= 64) return run_fwd<T, 64>(a, st);
  return run_fwd<T, 128>(a, st);
}

template <typename T>
int bwd_typed(const void* d_o, const void* q, const void* k, const void* v, const void* o, const float* row_max,
              const float* row_sum, void* dq, void* dk, void* dv, const int32_t* row_kstart, const ptj_attn_shape& sh,
              const ptj_attn_shape& dsh, const AttnDropout& dr, const unsigned int* patch, cudaStream_t st) {
  const void* ptrs[8] = {d_o, q, k, v, o, dq, dk, dv};
  const BwdArgs<T> a{static_cast<const T*>(d_o), static_cast<const T*>(q), static_cast<const T*>(k),
                     static_cast<const T*>(v), static_cast<const T*>(o), row_max, row_sum, static_cast<T*>(dq),
                     static_cast<T*>(dk), static_cast<T*>(dv), row_kstart, patch, sh, dsh,
                     1.f / sqrtf(static_cast<float>(sh.d_head)), static_cast<int>(ceil_div(sh.seq, kB)),
                     rows_vectorise<T>(sh, ptrs, 8) && rows_vectorise<T>(dsh, ptrs, 0), dr};
  if (sh.d_head <= 32) return run_bwd<T, 32>(a, st);
  if (sh.d_head <= 64) return run_bwd<T, 64>(a, st);
  return run_bwd<T, 128>(a, st);
}

}  // namespace

int attn_fwd_simt(const void* q, const void* k, const void* v, void* o, float* row_max, float* row_sum,
                  const int32_t* row_kstart, const ptj_attn_shape& sh, const AttnDropout& dr, int dtype, cudaStream_t st) {
  if (sh.d_head > kMaxD) return PTJ_ERR_UNSUPPORTED;
  return dtype == PTJ_F32 ? fwd_typed<float>(q, k, v, o, row_max, row_sum, row_kstart, sh, dr, st)
                          : fwd_typed<__nv_bfloat16>(q, k, v, o, row_max, row_sum, row_kstart, sh, dr, st);
}

int attn_bwd_simt(const void* d_o, const void* q, const void* k, const void* v, const void* o, const float* row_max,
                  const float* row_sum, void* dq, void* dk, void* dv, const int32_t* row_kstart,
                  const ptj_attn_shape& sh, const ptj_attn_shape& dsh, const AttnDropout& dr, int dtype,
                  const unsigned int* patch, cudaStream_t st) {
  if (sh.d_head > kMaxD) return PTJ_ERR_UNSUPPORTED;
  return dtype == PTJ_F32
             ? bwd_typed<float>(d_o, q, k, v, o, row_max, row_sum, dq, dk, dv, row_kstart, sh, dsh, dr, patch, st)
             : bwd_typed<__nv_bfloat16>(d_o, q, k, v, o, row_max, row_sum, dq, dk, dv, row_kstart, sh, dsh, dr, patch, st);
}

}  // namespace ptj
