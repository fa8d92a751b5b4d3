// Greedy decoding of a few sequences in one launch, float32 (loss_and_optimizer_triton.py:203-212 with train=False).
//
// The causal model's keys and values of earlier positions do not change when a token is appended, so a new token costs one
// row of every product: a pass over the weights, bound by reading them (4 bytes per parameter and token). One cooperative
// block per SM runs all tokens. Every matrix is a list of row pairs dealt to the blocks in contiguous ranges; a warp
// multiplies 128-wide chunks of a pair with the activations of all sequences, and a block finishes its own rows. Grid
// barriers separate the five steps of a layer (QKV, attention, out-projection, FFN-1, FFN-2) and the tokens.
//
// Which weights a warp reads next never depends on the activations, so its cp.async ring (DEPTH chunks of 1 KB) runs ahead
// through rows, steps, layers and tokens: memory stays busy while the block waits at a barrier, normalises or attends.
// A lane reads only bytes that it copied itself, so the ring needs no barrier.
//
// Measured, 12 layers x 768, vocabulary 35374, two sequences of 128: 38.4 ms, 302 us a token; the weights alone take 69 us,
// the rest is the chain of 61 steps (barrier, activations, normalisation, reduction). A whole forward pass per token on
// the tensor cores took 374 ms. 46.8 ms before these: the ring's next address kept in registers, layer pointers in shared
// memory (their loads stood in front of every unit), attention without block-wide scores, a barrier of one release and
// acquire without fences.
#include "common.cuh"
#include "tc_common.cuh"
#include "tc_runtime.h"

namespace ptj {
namespace {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kChunk = 128;  // floats of a row per chunk: 16 bytes per lane
constexpr int kSteps = 5;    // QKV, out-projection, FFN-1, FFN-2, LM head
constexpr int kMaxHead = 128;
constexpr int kLayerTensors = 10;  // g1, b1, w_qkv, w_o, g2, b2, w1, b1f, w2, b2f
constexpr int kSmemLimit = 227 * 1024;
constexpr unsigned int kFaultBarrier = 0x3101u, kFaultMisaligned = 0x3102u;

struct Step {
  int R, K;         // rows and row length of the matrix
  int nch;          // chunks of a row
  int cpp, parts;   // chunks per part of a row, parts: a warp takes (row pair, part)
};

struct DecodeParams {
  const float *w_emb, *b_head, *w_pos, *g_f, *b_f;
  const float* const* layers;  // [L][kLayerTensors]
  int B, V, D, L, H, F, S, start;
  float emb_scale, keep;       // sqrt(D); what evaluation multiplies every dropout site by
  Step step[kSteps];
  int act_ld;                  // floats of one sequence's activations in shared memory
  float *x, *q, *attn, *h, *kv;
  float* best;                 // [blocks][B] block maxima
  int* best_arg;
  int32_t* tokens;             // [B][S]
  unsigned int* barrier;       // zeroed
  unsigned int* fault;
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;  // 0: the destination is filled with zeros
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(n) : "memory");
}

// row pairs [first, first + n) of a step that this block owns
struct Share {
  int first, n;
};

// The order in which a warp meets the weights: (token, layer, step, unit, chunk). Between units a lane only moves a pointer:
// the ring is refilled in the multiplying loop, whose length is what the steps wait for.
struct Cursor {
  int t, l, s, u;
  int left, col, K;   // chunks of the unit still to fetch, this lane's column, row length
  const float* w;     // this lane's position in the pair's first row
  bool two, valid;
  const Share* share;
  const float* const* layers;  // in shared memory
  __device__ __forceinline__ void locate(const DecodeParams& p) {  // unit u of the current step, or the next step that has one
    while (u >= share[s].n * p.step[s].parts) {
      u = threadIdx.x >> 5;
      if (s == 4) {
        if (++t >= p.S - 1) {
          valid = false;
          return;
        }
        s = l = 0;
      } else if (s == 3) {
        if (l + 1 < p.L) {
          ++l;
          s = 0;
        } else {
          s = 4;
        }
      } else {
        ++s;
      }
    }
    const Step& st = p.step[s];
    const int pair = share[s].first + u / st.parts, c = u % st.parts * st.cpp;
    const int idx = s == 0 ? 2 : (s == 1 ? 3 : (s == 2 ? 6 : 8));
    K = st.K;
    col = c * kChunk + (threadIdx.x & 31) * 4;
    w = (s == 4 ? p.w_emb : layers[l * kLayerTensors + idx]) + static_cast<int64_t>(pair) * 2 * K + col;
    two = 2 * pair + 1 < st.R;
    left = min(st.nch - c, st.cpp);
  }
  __device__ __forceinline__ void init(const DecodeParams& p, const Share* sh, const float* const* lt) {
    share = sh;
    layers = lt;
    t = l = s = 0;
    u = threadIdx.x >> 5;
    valid = true;
    locate(p);
  }
};

// One ring slot: [2 rows][32 lanes] x 16 bytes. dst: this lane's place in the first row.
__device__ __forceinline__ void fetch(Cursor& cur, const DecodeParams& p, uint32_t dst) {
  if (cur.valid) {
    const bool in = cur.col < cur.K, in2 = in && cur.two;
    cp_async16(dst, in ? cur.w : p.w_emb, in);
    cp_async16(dst + 512, in2 ? cur.w + cur.K : p.w_emb, in2);
    cur.w += kChunk;
    cur.col += kChunk;
    if (--cur.left == 0) {
      cur.u += kWarps;
      cur.locate(p);
    }
  }
  cp_async_commit();  // one group per chunk, empty ones at the end: the wait below counts groups
}

// All blocks have arrived and their writes are visible. The wait is bounded; false: give up.
__device__ __forceinline__ bool grid_barrier(const DecodeParams& p, unsigned int& target, int* ok_s) {
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0) {
    asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(p.barrier) : "memory");
    const long long t0 = clock64();
    int ok = 1;
    unsigned int seen;
    for (;;) {
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(p.barrier) : "memory");
      if (static_cast<int>(seen - target) >= 0) break;
      if (clock64() - t0 > tc::kWaitLimitCycles) {
        tc::record_fault(p.fault, kFaultBarrier);
        ok = 0;
        break;
      }
    }
    *ok_s = ok;
  }
  __syncthreads();
  return *ok_s != 0;
}

// mean and reciprocal unbiased deviation (no epsilon, model_triton.py:1042-1080) of a row in shared memory, by one warp
__device__ __forceinline__ float2 warp_row_stats(const float* row, int D, int lane) {
  float s = 0.f;
#pragma unroll 4
  for (int i = lane * 4; i < D; i += 128) {
    const float4 v = *reinterpret_cast<const float4*>(row + i);
    s += (v.x + v.y) + (v.z + v.w);
  }
  const float mean = warp_sum(s) / static_cast<float>(D);
  float ss = 0.f;
#pragma unroll 4
  for (int i = lane * 4; i < D; i += 128) {
    const float4 v = *reinterpret_cast<const float4*>(row + i);
    const float a = v.x - mean, b = v.y - mean, c = v.z - mean, d = v.w - mean;
    ss += fmaf(a, a, b * b) + fmaf(c, c, d * d);
  }
  return make_float2(mean, 1.f / sqrtf(warp_sum(ss) / static_cast<float>(D - 1)));
}

// elements 4 i .. 4 i + 3 of a scale or shift; aligned: it starts on a 16-byte boundary
__device__ __forceinline__ float4 load_vector4(const float* v, int i, bool aligned) {
  if (aligned) return __ldg(reinterpret_cast<const float4*>(v) + i);
  return make_float4(__ldg(v + 4 * i), __ldg(v + 4 * i + 1), __ldg(v + 4 * i + 2), __ldg(v + 4 * i + 3));
}

struct Best {
  float v;
  int arg;
};
__device__ __forceinline__ Best better(Best a, Best b) {  // the larger value, the smaller index among equals
  return b.v > a.v || (b.v == a.v && b.arg < a.arg) ? b : a;
}

template <int NB, int DEPTH>
__global__ void __launch_bounds__(kThreads, 1)
decode_kernel(const __grid_constant__ DecodeParams p) {
  extern __shared__ __align__(16) uint8_t smem[];
  float* act = reinterpret_cast<float*>(smem + kWarps * DEPTH * 1024);  // [NB][act_ld], zero beyond the row
  const float** layers = reinterpret_cast<const float**>(act + NB * p.act_ld);  // [L][kLayerTensors]
  float* part = reinterpret_cast<float*>(layers + p.L * kLayerTensors);  // [units][2][NB]
  __shared__ int ok_s;
  __shared__ Share share[kSteps];
  __shared__ Best best_s[kWarps][NB];
  __shared__ int token_s[NB];
  __shared__ float2 stats_s[NB];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const uint32_t ring = tc::smem_u32(smem + warp * DEPTH * 1024) + lane * 16;
  const uint8_t* ring_p = smem + warp * DEPTH * 1024;

  if (tid < kSteps) {
    const int64_t pairs = (p.step[tid].R + 1) / 2;
    share[tid].first = static_cast<int>(pairs * blockIdx.x / gridDim.x);
    share[tid].n = static_cast<int>(pairs * (blockIdx.x + 1) / gridDim.x) - share[tid].first;
  }
  if (tid < p.B) token_s[tid] = p.start;
  // The host cannot see these pointers. Matrices are copied in 16-byte pieces; scales and shifts may lie on any float.
  auto off16 = [](const float* q) { return (reinterpret_cast<uintptr_t>(q) & 15u) != 0; };
  bool bad = false, odd = off16(p.g_f) || off16(p.b_f);
  for (int i = tid; i < p.L * kLayerTensors; i += kThreads) {
    layers[i] = p.layers[i];
    const int k = i % kLayerTensors;
    (k == 2 || k == 3 || k == 6 || k == 8 ? bad : odd) |= off16(layers[i]);
  }
  if (__syncthreads_or(bad)) {  // the same in every block: none waits for another yet
    if (blockIdx.x == 0 && tid == 0) tc::record_fault(p.fault, kFaultMisaligned);
    return;
  }
  const bool aligned = !__syncthreads_or(odd);
  Cursor cur;
  cur.init(p, share, layers);
#pragma unroll 1
  for (int i = 0; i < DEPTH - 1; ++i) fetch(cur, p, ring + i * 1024);
  int slot = 0;                     // next chunk to consume
  int free_slot = DEPTH - 1;        // next slot to fill
  unsigned int target = 0;
  const int dh = p.D / p.H;
  const int64_t kv_plane = static_cast<int64_t>(p.S) * dh;  // one sequence's, head's and layer's keys (or values)


  // this block's share of a step's products: partial sums of unit u, row r, sequence b at part[(u * 2 + r) * NB + b]
  auto multiply = [&](int s) {
    const Step& st = p.step[s];
    const int nunits = share[s].n * st.parts;
    for (int u = warp; u < nunits; u += kWarps) {
      const int c0 = u % st.parts * st.cpp, c1 = min(st.nch, c0 + st.cpp);
      float acc[2][NB];
#pragma unroll
      for (int b = 0; b < NB; ++b) acc[0][b] = acc[1][b] = 0.f;
      for (int c = c0; c < c1; ++c) {
        cp_async_wait<DEPTH - 2>();
        const float4 w0 = *reinterpret_cast<const float4*>(ring_p + slot * 1024 + lane * 16);
        const float4 w1 = *reinterpret_cast<const float4*>(ring_p + slot * 1024 + 512 + lane * 16);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const float4 a = *reinterpret_cast<const float4*>(act + b * p.act_ld + c * kChunk + lane * 4);
          acc[0][b] = fmaf(w0.w, a.w, fmaf(w0.z, a.z, fmaf(w0.y, a.y, fmaf(w0.x, a.x, acc[0][b]))));
          acc[1][b] = fmaf(w1.w, a.w, fmaf(w1.z, a.z, fmaf(w1.y, a.y, fmaf(w1.x, a.x, acc[1][b]))));
        }
        fetch(cur, p, ring + free_slot * 1024);
        slot = slot + 1 == DEPTH ? 0 : slot + 1;
        free_slot = free_slot + 1 == DEPTH ? 0 : free_slot + 1;
      }
#pragma unroll
      for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int b = 0; b < NB; ++b) {
          const float v = warp_sum(acc[r][b]);
          if (lane == r * NB + b) part[(u * 2 + r) * NB + b] = v;
        }
    }
    __syncthreads();
  };
  // The products of a step and finish(row, b, sum, side(row, b)) for every output of this block's rows. side (a bias and the
  // residual) is read from memory before the products for the first output of a thread, which is the only one as a rule.
  auto run_step = [&](int s, auto&& side, auto&& finish) {
    const Step& st = p.step[s];
    const int row0 = 2 * share[s].first, n = share[s].n * 2 * NB;
    auto real = [&](int i) { return i < n && i % NB < p.B && row0 + i / NB < st.R; };
    const float2 side0 = real(tid) ? side(row0 + tid / NB, tid % NB) : make_float2(0.f, 0.f);
    multiply(s);
    for (int i = tid; i < n; i += kThreads) {
      if (!real(i)) continue;
      const int b = i % NB, rr = i / NB;
      float v = 0.f;
      for (int k = 0; k < st.parts; ++k) v += part[(((rr >> 1) * st.parts + k) * 2 + (rr & 1)) * NB + b];
      finish(row0 + rr, b, v, i == tid ? side0 : side(row0 + rr, b));
    }
  };
  auto load_act = [&](const float* src, int K) {  // [B][K] written by other blocks
    for (int b = 0; b < p.B; ++b)
      for (int i = tid * 4; i < K; i += kThreads * 4)
        *reinterpret_cast<float4*>(act + b * p.act_ld + i) = __ldcg(reinterpret_cast<const float4*>(src + b * K + i));
  };
  // a step reads K columns; what an earlier, longer row left in its last chunk would meet zero weights, which infinities
  // and NaNs survive: cleared
  auto clear_tail = [&](const Step& st) {
    const int n = st.nch * kChunk - st.K;
    for (int i = tid; i < n * NB; i += kThreads) act[i / n * p.act_ld + st.K + i % n] = 0.f;
  };
  // LayerNorm of the B rows in shared memory: a warp per row for the statistics, all threads for the elements. Scale and
  // shift of a thread's first four elements are on their way while the statistics are formed.
  auto normalise = [&](const float* g, const float* b) {
    const int nd = p.D / 4, n = p.B * nd;
    float4 g0, b0;
    if (tid < n) {
      g0 = load_vector4(g, tid % nd, aligned);
      b0 = load_vector4(b, tid % nd, aligned);
    }
    __syncthreads();
    if (warp < p.B) {
      const float2 st = warp_row_stats(act + warp * p.act_ld, p.D, lane);
      if (lane == 0) stats_s[warp] = st;
    }
    __syncthreads();
    for (int i = tid; i < n; i += kThreads) {
      if (i != tid) {
        g0 = load_vector4(g, i % nd, aligned);
        b0 = load_vector4(b, i % nd, aligned);
      }
      const float2 st = stats_s[i / nd];
      float4* x = reinterpret_cast<float4*>(act + i / nd * p.act_ld) + i % nd;
      float4 v = *x;
      v.x = g0.x * ((v.x - st.x) * st.y) + b0.x;
      v.y = g0.y * ((v.y - st.x) * st.y) + b0.y;
      v.z = g0.z * ((v.z - st.x) * st.y) + b0.z;
      v.w = g0.w * ((v.w - st.x) * st.y) + b0.w;
      *x = v;
    }
    __syncthreads();
  };
  const auto none = [](int, int) { return make_float2(0.f, 0.f); };

  for (int pos = 0; pos < p.S - 1; ++pos) {
    // embedding of the token at `pos`: every block forms the whole row, and keeps its own rows of the residual stream
    const int x0 = 2 * share[1].first, x1 = x0 + 2 * share[1].n;
    for (int i = tid; i < p.B * p.D; i += kThreads) {
      const int b = i / p.D, d = i - b * p.D;
      const int tok = min(max(token_s[b], 0), p.V - 1);
      const float e = (p.w_emb[static_cast<int64_t>(tok) * p.D + d] * p.emb_scale + p.w_pos[static_cast<int64_t>(pos) * p.D + d]) * p.keep;
      act[b * p.act_ld + d] = e;
      if (d >= x0 && d < x1) p.x[i] = e;
    }
    for (int l = 0; l < p.L; ++l) {
      const float* const* w = layers + l * kLayerTensors;
      float* kv = p.kv + static_cast<int64_t>(l) * p.B * p.H * 2 * kv_plane;
      // QKV: rows ordered (head, q/k/v, d)
      if (l > 0) load_act(p.x, p.D);
      clear_tail(p.step[0]);
      normalise(w[0], w[1]);
      run_step(0, none, [&](int row, int b, float v, float2) {
        const int hd = row / (3 * dh), c = row / dh % 3, d = row % dh;
        if (c == 0) p.q[(b * p.H + hd) * dh + d] = v;
        else kv[((static_cast<int64_t>(b) * p.H + hd) * 2 + (c - 1)) * kv_plane + static_cast<int64_t>(pos) * dh + d] = v;
      });
      if (!grid_barrier(p, target, &ok_s)) goto out;

      // attention of one position over the cached keys: a block per (sequence, head)
      {
        // A group of lanes takes every groups-th key with a running maximum, sum and output of its own, so that no thread
        // waits for another before the groups are merged.
        int lpk = 1;  // lanes per key
        while (lpk * 4 < dh) lpk *= 2;
        const int sub = lane % lpk, group = tid / lpk, groups = kThreads / lpk;
        const bool on = sub * 4 < dh;
        float* red = act;        // [groups][dh] outputs
        float* ml = part;        // [groups][2] maxima, sums
        const float scale = 1.f / sqrtf(static_cast<float>(dh));
        for (int bh = blockIdx.x; bh < p.B * p.H; bh += gridDim.x) {
          const float* kb = kv + static_cast<int64_t>(bh) * 2 * kv_plane + sub * 4;
          const float* vb = kb + kv_plane;
          const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
          const float4 q = on ? __ldcg(reinterpret_cast<const float4*>(p.q + bh * dh + sub * 4)) : zero;
          float m = -INFINITY, sum = 0.f;
          float4 o = zero;
          for (int j0 = 0; j0 <= pos; j0 += 4 * groups) {
            float4 k[4], v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int j = j0 + e * groups + group;
              const bool in = on && j <= pos;
              k[e] = in ? __ldcg(reinterpret_cast<const float4*>(kb + static_cast<int64_t>(j) * dh)) : zero;
              v[e] = in ? __ldcg(reinterpret_cast<const float4*>(vb + static_cast<int64_t>(j) * dh)) : zero;
            }
            float s[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) s[e] = fmaf(q.x, k[e].x, fmaf(q.y, k[e].y, fmaf(q.z, k[e].z, q.w * k[e].w)));
            for (int x = lpk / 2; x > 0; x >>= 1) {
#pragma unroll
              for (int e = 0; e < 4; ++e) s[e] += __shfl_xor_sync(0xffffffffu, s[e], x);
            }
            float mnew = m;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              s[e] = j0 + e * groups + group <= pos ? s[e] * scale : -INFINITY;
              mnew = fmaxf(mnew, s[e]);
            }
            const float ref = mnew == -INFINITY ? 0.f : mnew;
            const float corr = expf(m - ref);
            sum *= corr;
            o.x *= corr; o.y *= corr; o.z *= corr; o.w *= corr;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const float pe = expf(s[e] - ref);
              sum += pe;
              o.x = fmaf(pe, v[e].x, o.x); o.y = fmaf(pe, v[e].y, o.y); o.z = fmaf(pe, v[e].z, o.z); o.w = fmaf(pe, v[e].w, o.w);
            }
            m = mnew;
          }
          if (on) *reinterpret_cast<float4*>(red + group * dh + sub * 4) = o;
          if (sub == 0) {
            ml[2 * group] = m;
            ml[2 * group + 1] = sum;
          }
          __syncthreads();
          if (tid < dh) {
            const int n = min(groups, pos + 1);  // the groups that hold keys
            float mm = -INFINITY, l = 0.f, v = 0.f;
#pragma unroll 8
            for (int g = 0; g < n; ++g) mm = fmaxf(mm, ml[2 * g]);
#pragma unroll 8
            for (int g = 0; g < n; ++g) {
              const float f = expf(ml[2 * g] - mm);
              l = fmaf(f, ml[2 * g + 1], l);
              v = fmaf(f, red[g * dh + tid], v);
            }
            p.attn[bh * dh + tid] = v * (p.keep / l);  // heads are consecutive: [B][D]
          }
          __syncthreads();
        }
      }
      if (!grid_barrier(p, target, &ok_s)) goto out;

      load_act(p.attn, p.D);
      clear_tail(p.step[1]);
      __syncthreads();
      run_step(1, [&](int row, int b) { return make_float2(0.f, p.x[b * p.D + row]); },
               [&](int row, int b, float v, float2 e) { p.x[b * p.D + row] = fmaf(v, p.keep, e.y); });
      if (!grid_barrier(p, target, &ok_s)) goto out;

      load_act(p.x, p.D);
      clear_tail(p.step[2]);
      normalise(w[4], w[5]);
      run_step(2, [&](int row, int) { return make_float2(__ldg(w[7] + row), 0.f); },
               [&](int row, int b, float v, float2 e) { p.h[b * p.F + row] = gelu_tanh(v + e.x); });
      if (!grid_barrier(p, target, &ok_s)) goto out;

      load_act(p.h, p.F);
      clear_tail(p.step[3]);
      __syncthreads();
      run_step(3, [&](int row, int b) { return make_float2(__ldg(w[9] + row), p.x[b * p.D + row]); },
               [&](int row, int b, float v, float2 e) { p.x[b * p.D + row] = fmaf(v + e.x, p.keep, e.y); });
      if (!grid_barrier(p, target, &ok_s)) goto out;
    }

    // LM head and arg-max
    load_act(p.x, p.D);
    clear_tail(p.step[4]);
    normalise(p.g_f, p.b_f);
    Best mine[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) mine[b] = Best{-INFINITY, 0x7fffffff};
    run_step(4, [&](int row, int) { return make_float2(__ldg(p.b_head + row), 0.f); }, [&](int row, int b, float v, float2 e) {
      const Best c{v + e.x, row};
#pragma unroll
      for (int k = 0; k < NB; ++k)
        if (k == b) mine[k] = better(mine[k], c);
    });
    // (a row without any value above -inf takes the index 0, as torch.argmax does)
    auto warp_best = [&](Best v) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
        v = better(v, Best{__shfl_xor_sync(0xffffffffu, v.v, o), __shfl_xor_sync(0xffffffffu, v.arg, o)});
      return v;
    };
#pragma unroll
    for (int b = 0; b < NB; ++b) {
      const Best v = warp_best(mine[b]);
      if (lane == 0) best_s[warp][b] = v;
    }
    __syncthreads();
    if (tid < p.B) {
      Best v = best_s[0][tid];
      for (int k = 1; k < kWarps; ++k) v = better(v, best_s[k][tid]);
      p.best[blockIdx.x * p.B + tid] = v.v;
      p.best_arg[blockIdx.x * p.B + tid] = v.arg;
    }
    if (!grid_barrier(p, target, &ok_s)) goto out;
    if (warp < p.B) {
      Best v{-INFINITY, 0x7fffffff};
      for (int k = lane; k < static_cast<int>(gridDim.x); k += 32)
        v = better(v, Best{__ldcg(p.best + k * p.B + warp), __ldcg(p.best_arg + k * p.B + warp)});
      v = warp_best(v);
      if (lane == 0) {
        const int tok = v.v == -INFINITY ? 0 : v.arg;
        token_s[warp] = tok;
        if (blockIdx.x == 0) p.tokens[warp * p.S + pos + 1] = tok;
      }
    }
    __syncthreads();  // (the next token overwrites p.best only after the barriers of its layers)
  }
out:
  cp_async_wait<0>();
}

Step make_step(int R, int K) {
  Step s;
  s.R = R;
  s.K = K;
  s.nch = (K + kChunk - 1) / kChunk;
  const int pairs_per_block = static_cast<int>(ceil_div((R + 1) / 2, kNumSMs));
  int want = kWarps / pairs_per_block;  // short lists of rows are cut along the row, so that all warps of a block have work
  if (want < 1) want = 1;
  if (want > s.nch) want = s.nch;
  s.cpp = (s.nch + want - 1) / want;
  s.parts = (s.nch + s.cpp - 1) / s.cpp;
  return s;
}

struct Plan {
  DecodeParams p;
  int nb, depth;
  size_t smem;
  size_t kv_floats, floats;  // workspace: kv, x, q, attn, h, best, best_arg, barrier
};

constexpr int kDepths[3] = {12, 8, 5};

bool make_plan(int64_t B, int64_t V, int64_t D, int64_t L, int64_t H, int64_t F, int64_t S, Plan& out) {
  if (B < 1 || B > 8 || V < 1 || D < 8 || L < 1 || H < 1 || F < 4 || S < 2) return false;
  if (D % H != 0 || D % 4 != 0 || F % 4 != 0 || (D / H) % 4 != 0 || D / H > kMaxHead) return false;
  if (V > (1 << 24) || D > (1 << 16) || F > (1 << 18) || S > 16384 || L > 4096) return false;
  DecodeParams& p = out.p;
  p = DecodeParams{};
  p.B = static_cast<int>(B); p.V = static_cast<int>(V); p.D = static_cast<int>(D); p.L = static_cast<int>(L);
  p.H = static_cast<int>(H); p.F = static_cast<int>(F); p.S = static_cast<int>(S);
  p.step[0] = make_step(3 * p.D, p.D);
  p.step[1] = make_step(p.D, p.D);
  p.step[2] = make_step(p.F, p.D);
  p.step[3] = make_step(p.D, p.F);
  p.step[4] = make_step(p.V, p.D);
  out.nb = B <= 1 ? 1 : (B <= 2 ? 2 : (B <= 4 ? 4 : 8));
  int units = 0, ld = 0;
  for (const Step& s : p.step) {
    const int u = static_cast<int>(ceil_div((s.R + 1) / 2, kNumSMs)) * s.parts;
    units = u > units ? u : units;
    ld = s.nch * kChunk > ld ? s.nch * kChunk : ld;
  }
  // the attention step keeps its groups' maxima and sums where the partial sums go, and their outputs where the
  // activations go
  int lpk = 1;
  while (lpk * 4 < p.D / p.H) lpk *= 2;
  const int red = kThreads / lpk * (p.D / p.H);
  size_t part = static_cast<size_t>(units) * 2 * out.nb;
  if (part < static_cast<size_t>(2 * kThreads / lpk)) part = 2 * kThreads / lpk;
  if (ld * out.nb < red) ld = static_cast<int>(ceil_div(ceil_div(red, out.nb), 4) * 4);
  p.act_ld = ld;
  const size_t fixed = (static_cast<size_t>(ld) * out.nb + part) * 4 + static_cast<size_t>(L) * kLayerTensors * 8;
  out.depth = 0;
  for (int d : kDepths) {
    out.smem = static_cast<size_t>(kWarps) * d * 1024 + fixed;
    if (out.smem + 2048 <= kSmemLimit) {  // (static shared memory: block maxima, shares, tokens)
      out.depth = d;
      break;
    }
  }
  if (out.depth == 0) return false;
  out.kv_floats = static_cast<size_t>(L) * B * H * 2 * S * (D / H);
  out.floats = out.kv_floats + static_cast<size_t>(B) * (3 * D + F) + 2 * static_cast<size_t>(kNumSMs) * B + 32;
  return true;
}

template <int NB, int DEPTH>
int launch(const Plan& pl, cudaStream_t st) {
  auto kern = decode_kernel<NB, DEPTH>;
  int blocks = 0;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(pl.smem)) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kern, kThreads, pl.smem) != cudaSuccess || blocks < 1) {
    (void)cudaGetLastError();
    return PTJ_ERR_LAUNCH;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(kNumSMs);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = pl.smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;  // the blocks wait for one another: all are resident or none starts
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (cudaLaunchKernelEx(&cfg, kern, pl.p) != cudaSuccess) {
    (void)cudaGetLastError();
    return PTJ_ERR_LAUNCH;
  }
  count_launch(1);
  return PTJ_OK;
}
template <int NB>
int launch_depth(const Plan& pl, cudaStream_t st) {
  return pl.depth == 12 ? launch<NB, 12>(pl, st) : (pl.depth == 8 ? launch<NB, 8>(pl, st) : launch<NB, 5>(pl, st));
}

}  // namespace
}  // namespace ptj

using namespace ptj;

extern "C" size_t ptj_decode_workspace_floats(int64_t batch, int64_t vocab, int64_t dim, int64_t layers, int64_t heads,
                                              int64_t ffn, int64_t seq) {
  Plan pl;
  return make_plan(batch, vocab, dim, layers, heads, ffn, seq, pl) ? pl.floats : 0;
}

extern "C" int ptj_decode(const float* w_emb, const float* b_head, const float* w_pos, const float* const* layer_tensors,
                          const float* g_f, const float* b_f, int32_t* tokens, int64_t start, float p, int64_t batch,
                          int64_t vocab, int64_t dim, int64_t layers, int64_t heads, int64_t ffn, int64_t seq,
                          float* workspace, size_t workspace_floats, void* stream) {
  Plan pl;
  if (!w_emb || !b_head || !w_pos || !layer_tensors || !g_f || !b_f || !tokens || !(p >= 0.f && p <= 1.f))
    return PTJ_ERR_BAD_SHAPE;
  if (!make_plan(batch, vocab, dim, layers, heads, ffn, seq, pl)) return PTJ_ERR_UNSUPPORTED;
  if (workspace == nullptr || workspace_floats < pl.floats) return PTJ_ERR_WORKSPACE;
  if (!aligned16(w_emb) || !aligned16(workspace)) return PTJ_ERR_MISALIGNED;
  if (ptj_device_check() != PTJ_OK) return PTJ_ERR_DEVICE;
  DecodeParams& d = pl.p;
  d.w_emb = w_emb; d.b_head = b_head; d.w_pos = w_pos; d.g_f = g_f; d.b_f = b_f;
  d.layers = layer_tensors;
  d.tokens = tokens;
  d.start = static_cast<int>(start < 0 ? 0 : (start >= vocab ? vocab - 1 : start));
  d.emb_scale = sqrtf(static_cast<float>(dim));
  d.keep = 1.f - p;
  float* ws = workspace;
  d.kv = ws; ws += pl.kv_floats;
  d.x = ws; ws += batch * dim;
  d.q = ws; ws += batch * dim;
  d.attn = ws; ws += batch * dim;
  d.h = ws; ws += batch * ffn;
  d.barrier = reinterpret_cast<unsigned int*>(ws); ws += 32;
  d.best = ws; ws += kNumSMs * batch;
  d.best_arg = reinterpret_cast<int*>(ws);
  d.fault = tc::fault_word();
  if (d.fault == nullptr) return PTJ_ERR_DEVICE;
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(d.barrier, 0, 4, st) != cudaSuccess) {
    (void)cudaGetLastError();
    return PTJ_ERR_LAUNCH;
  }
  switch (pl.nb) {
    case 1: return launch_depth<1>(pl, st);
    case 2: return launch_depth<2>(pl, st);
    case 4: return launch_depth<4>(pl, st);
    default: return launch_depth<8>(pl, st);
  }
}
