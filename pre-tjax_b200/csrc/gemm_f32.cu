// float32 GEMM on the tensor cores.
//
// Every float32 operand element a, times 2^24, is split exactly into three bf16 values, 2^24 a = a1 + a2 + a3 (8 + 8 + 8
// mantissa bits, round to nearest), and the product is the sum of the six partial products whose magnitude can matter in float32:
//   a1 b1 + (a1 b2 + a2 b1) + (a2 b2 + a1 b3 + a3 b1);   what is left out is below 2^-26 of |a b|.
// The factor keeps the last bits of the smallest numbers (multiples of 2^-149) above bf16's smallest normal value, 2^-126;
// without it parts of elements below 2^-110 were lost. 2^-48 times the sum undoes it, exactly down to float32's subnormals.
// bf16 products are exact in the tensor core; its float32 accumulator, however, truncates at every step of an
// accumulation chain, which over a long K would bias the result. So a chain is only 64 elements of K long, runs from the
// smallest partial products to the largest (four truncations at full magnitude), and the epilogue warps add each
// finished chain into float32 REGISTERS with round-to-nearest. Measured against float64 the result is as accurate as a
// sequential fused-multiply-add loop or better (tests/test_gemm_f32_gpu.py compares the two). Operands with infinities, or
// so large that a partial product could overflow, are found by the splitting pass and take the fused-multiply-add loop.
//
// Two launches: a splitting pass writes the three bf16 planes of both operands ([3][rows][ld], same storage order as the
// operand, so K-major and MN-major operands need no transposition), then a persistent thread-block-pair kernel like the
// bf16 one multiplies 256 x 256 tiles. One 64-deep stage of K brings 3 planes x (128 + 128) rows x 128 bytes = 96 KB per
// CTA, from which 24 MMAs of 256 x 256 x 16 are issued (3 072 clk): 32 B/clk/SM of operands, half of what the bf16
// kernel needs per MMA, so the tensor pipe and not the L2 feed bounds it. Two such stages fill shared memory.
//
// Measured (B200): 240 TFLOP/s of float32 product at [4096, 35376] x 768 (1.44 PFLOP/s of bf16 MMAs), 198 at [4096, 2304] x
// 768, both including the splitting pass; the kernel this replaces there ran at 24. More sizes beside use_f32_tc().
#include <atomic>

#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "gemm_f32.h"
#include "tc_common.cuh"
#include "tc_runtime.h"

namespace ptj {
namespace {

using namespace tc;

constexpr int BM = 128, BN = 256, BK = 64, HB = BN / 2;
constexpr int kPlaneBytes = 128 * BK * 2;             // one plane of one operand half: 128 rows x 64 columns
constexpr int kOperandBytes = 3 * kPlaneBytes;        // 48 KB
constexpr int kStageBytes = 2 * kOperandBytes;
constexpr int kStages = 2;
constexpr int kEpilogueWarps = 8, kFirstEpilogueWarp = 4;
constexpr int kThreads = 32 * (kFirstEpilogueWarp + kEpilogueWarps);
// (4 x 40 + 8 x 232) x 32 registers fit the block's 384 x 168: the epilogue warps keep 128 accumulators per thread
constexpr int kRegsIssue = 40, kRegsEpilogue = 232;
constexpr int kSmemBytes = kStages * kStageBytes + kEpilogueWarps * kStripBytes + 1024 + 256;
static_assert(kSmemBytes <= 227 * 1024, "shared memory of one block");
constexpr int kPairs = kNumSMs / 2;

struct F32Params {
  EpilogueParams ep;
  int64_t M, N;
  int num_m, num_n, num_kb, split_k;
  float* workspace;  // [split_k, M, N] partial sums when split_k > 1
  // the operands themselves, for products with elements that the parts cannot carry
  const float *a, *b;
  int64_t lda, ldb, K;
  const int* flags;  // [num_flags] one per block of the splitting pass: it met such an element
  int num_flags;
  int* any_flag;     // whether any is set, for the finishing kernel
  unsigned int* fault;
};

// Operands with an infinity, or with a finite magnitude of 2^24 or more, are multiplied by fused multiply-adds instead, as if
// there were no tensor-core path: an infinity times the parts of a number gives NaNs (their signs differ, or they are zero),
// and products of parts may overflow where the sum does not. Below 2^24 neither can happen: the sum of products of scaled
// elements, each below 2^48, stays below 2^30 2^96.
constexpr float kBig = 16777216.f, kScale = 16777216.f;  // 2^24 both
constexpr float kUnscale = 1.f / (kScale * kScale);

// ---- splitting pass -------------------------------------------------------------------------------------------------
struct SplitSrc {
  const float* src;
  __nv_bfloat16* dst;  // [3][rows][ldp]
  int64_t ld, rows, cols, ldp;
};

__device__ __forceinline__ void split3(float x, uint16_t& p1, uint16_t& p2, uint16_t& p3) {
  const float a = x * kScale;
  const __nv_bfloat16 h1 = __float2bfloat16_rn(a);
  const float r1 = isnan(a) ? 0.f : a - __bfloat162float(h1);  // exact; a NaN goes through alone
  const __nv_bfloat16 h2 = __float2bfloat16_rn(r1);
  const float r2 = r1 - __bfloat162float(h2);  // exact, at most eight significant bits
  p1 = __bfloat16_as_ushort(h1);
  p2 = __bfloat16_as_ushort(h2);
  p3 = __bfloat16_as_ushort(__float2bfloat16_rn(r2));
}

// Memory-bound: 4 bytes read and 6 written per element, eight elements per thread.
__global__ void __launch_bounds__(256)
split_planes_kernel(const SplitSrc s0, const SplitSrc s1, int* __restrict__ flags) {
  grid_dep_sync();
  float top = 0.f;  // largest magnitude, NaNs aside
  const int64_t g0 = s0.rows * (s0.ldp / 8), total = g0 + s1.rows * (s1.ldp / 8);
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const bool second = i >= g0;
    const SplitSrc& s = second ? s1 : s0;
    const int64_t li = second ? i - g0 : i;
    const int64_t groups = s.ldp / 8, r = li / groups, c = (li - r * groups) * 8;
    const float* src = s.src + r * s.ld + c;
    float v[8];
    if (c + 8 <= s.cols && (reinterpret_cast<uintptr_t>(src) & 15u) == 0) {
      const float4 a = __ldg(reinterpret_cast<const float4*>(src)), b = __ldg(reinterpret_cast<const float4*>(src) + 1);
      v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w; v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
    } else {
#pragma unroll
      for (int j = 0; j < 8; ++j) v[j] = c + j < s.cols ? src[j] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) top = fmaxf(top, fabsf(v[j]));
    uint32_t w[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint16_t lo[3], hi[3];
      split3(v[2 * j], lo[0], lo[1], lo[2]);
      split3(v[2 * j + 1], hi[0], hi[1], hi[2]);
#pragma unroll
      for (int p = 0; p < 3; ++p) w[p][j] = static_cast<uint32_t>(lo[p]) | (static_cast<uint32_t>(hi[p]) << 16);
    }
    const int64_t plane = s.rows * s.ldp;
#pragma unroll
    for (int p = 0; p < 3; ++p)
      *reinterpret_cast<uint4*>(s.dst + p * plane + r * s.ldp + c) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
  }
  const int any = __syncthreads_or(top >= kBig);
  if (threadIdx.x == 0) flags[blockIdx.x] = any;
}

// ---- product --------------------------------------------------------------------------------------------------------

__device__ __forceinline__ void epilogue_warps_sync() { asm volatile("barrier.sync 1, %0;" ::"n"(kEpilogueWarps * 32) : "memory"); }

// The whole product by fused multiply-adds, in the order of the kernel in gemm.cu (one sum per output, along K): the same
// bits. Run by the epilogue warps in their store strips: 64 x 128 outputs a block, 4 x 8 a thread; the next 16 of K are on
// their way while a tile of them is multiplied. [4096, 2304] x 768 with one infinity: 591 us (72 without, 593 on the kernel in
// gemm.cu); [256, 256] x 256: 110 us (20, 20), as the launch has the few blocks that the tensor-core tiles need. Not inlined:
// as part of the kernel it took registers from the epilogue ([4096, 2304] x 768 without an infinity: 76 us).
constexpr int kFmaM = 64, kFmaN = 128, kFmaK = 16;
constexpr int kFmaLdA = kFmaM + 4, kFmaLdB = kFmaN + 4;
static_assert(kEpilogueWarps * 32 == (kFmaM / 4) * (kFmaN / 8), "a thread per 4 x 8 outputs");
static_assert(kFmaK * (kFmaLdA + kFmaLdB) * 4 <= kEpilogueWarps * kStripBytes, "operand tiles fit the strips");
template <bool A_KMAJOR, bool B_KMAJOR>
__device__ __noinline__ void product_by_fma(const F32Params& p, float* smem, uint64_t seed, int tid) {
  constexpr int kN = kEpilogueWarps * 32, kA = kFmaM * kFmaK / kN, kB = kFmaN * kFmaK / kN;
  float* a_s = smem;                     // [kFmaK][kFmaLdA]
  float* b_s = smem + kFmaK * kFmaLdA;   // [kFmaK][kFmaLdB]: columns 8 x + 4 h + e at 64 h + 4 x + e, read without conflicts
  const int tx = tid % (kFmaN / 8), ty = tid / (kFmaN / 8);
  const int64_t M = p.M, N = p.N, K = p.K, lda = p.lda, ldb = p.ldb;
  const float *A = p.a, *B = p.b;
  const int64_t cols = (N + kFmaN - 1) / kFmaN, tiles = (M + kFmaM - 1) / kFmaM * cols;
  for (int64_t tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    const int64_t m0 = tile / cols * kFmaM, n0 = tile % cols * kFmaN;
    float ra[kA], rb[kB], acc[4][8];
    auto fetch = [&](int64_t k0) {
#pragma unroll
      for (int e = 0; e < kA; ++e) {
        const int i = tid + e * kN, r = A_KMAJOR ? i / kFmaK : i % kFmaM, k = A_KMAJOR ? i % kFmaK : i / kFmaM;
        const int64_t m = m0 + r, kk = k0 + k;
        ra[e] = m < M && kk < K ? A[A_KMAJOR ? m * lda + kk : kk * lda + m] : 0.f;
      }
#pragma unroll
      for (int e = 0; e < kB; ++e) {
        const int i = tid + e * kN, r = B_KMAJOR ? i / kFmaK : i % kFmaN, k = B_KMAJOR ? i % kFmaK : i / kFmaN;
        const int64_t n = n0 + r, kk = k0 + k;
        rb[e] = n < N && kk < K ? B[B_KMAJOR ? n * ldb + kk : kk * ldb + n] : 0.f;
      }
    };
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = 0.f;
    fetch(0);
    for (int64_t k0 = 0; k0 < K; k0 += kFmaK) {
      epilogue_warps_sync();  // the tile before has been read
#pragma unroll
      for (int e = 0; e < kA; ++e) {
        const int i = tid + e * kN, r = A_KMAJOR ? i / kFmaK : i % kFmaM, k = A_KMAJOR ? i % kFmaK : i / kFmaM;
        a_s[k * kFmaLdA + r] = ra[e];
      }
#pragma unroll
      for (int e = 0; e < kB; ++e) {
        const int i = tid + e * kN, r = B_KMAJOR ? i / kFmaK : i % kFmaN, k = B_KMAJOR ? i % kFmaK : i / kFmaN;
        b_s[k * kFmaLdB + (r % 8 / 4) * (kFmaN / 2) + r / 8 * 4 + r % 4] = rb[e];
      }
      epilogue_warps_sync();
      if (k0 + kFmaK < K) fetch(k0 + kFmaK);
#pragma unroll 4
      for (int k = 0; k < kFmaK; ++k) {
        const float4 a = *reinterpret_cast<const float4*>(a_s + k * kFmaLdA + ty * 4);
        const float4 b0 = *reinterpret_cast<const float4*>(b_s + k * kFmaLdB + tx * 4);
        const float4 b1 = *reinterpret_cast<const float4*>(b_s + k * kFmaLdB + kFmaN / 2 + tx * 4);
        const float av[4] = {a.x, a.y, a.z, a.w}, bv[8] = {b0.x, b0.y, b0.z, b0.w, b1.x, b1.y, b1.z, b1.w};
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) epilogue_row_segment<float, 8>(p.ep, m0 + ty * 4 + i, n0 + tx * 8, acc[i], seed);
  }
}

template <bool A_KMAJOR, bool B_KMAJOR>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_pair_kernel(const __grid_constant__ CUtensorMap tmap_a, const __grid_constant__ CUtensorMap tmap_b,
                     const __grid_constant__ F32Params p) {
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
  uint8_t* strips = smem + kStages * kStageBytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(strips + kEpilogueWarps * kStripBytes);  // used in the leader only
  uint64_t* empty = full + kStages;       // one set per CTA, both signalled by the leader's commits
  uint64_t* tmem_full = empty + kStages;
  uint64_t* tmem_empty = tmem_full + 2;   // used in the leader only: 8 local + 8 remote epilogue warps
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tmem_empty + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* epi_state = reinterpret_cast<int*>(tmem_slot + 2);  // written by the epilogue warps: 1 multiply by FMA, 2 a wait ran out

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = cluster_ctarank();
  const AbortCtx ctx{abort_flag, p.fault};

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&tmem_full[b], 1);
      mbar_init(&tmem_empty[b], 2 * kEpilogueWarps);
    }
    *abort_flag = 0;
    *epi_state = 0;
    fence_barrier_init();
    prefetch_tensormap(&tmap_a);
    prefetch_tensormap(&tmap_b);
  }
  __syncthreads();
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, 512);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers are initialised before anyone signals across the pair
  tc_fence_after_sync();
  grid_dep_sync();
  const uint32_t tmem_base = *tmem_slot;

  const int tiles = p.num_m * p.num_n, total = tiles * p.split_k;
  const int pair = static_cast<int>(blockIdx.x) >> 1, npairs = static_cast<int>(gridDim.x) >> 1;
  if (warp < kFirstEpilogueWarp) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIssue));

  if (warp == 0) {
    if (lane == 0) {
      int stage = 0;
      uint32_t phase = 0;
      bool ok = true;
      for (int item = pair; item < total && ok; item += npairs) {
        const int split = item / tiles, tile = item - split * tiles;
        const int m_blk = tile % p.num_m, n_blk = tile / p.num_m;
        const int kb0 = static_cast<int>(static_cast<int64_t>(split) * p.num_kb / p.split_k);
        const int kb1 = static_cast<int>(static_cast<int64_t>(split + 1) * p.num_kb / p.split_k);
        const int m0 = m_blk * 2 * BM + static_cast<int>(rank) * BM;
        const int n0 = n_blk * BN + static_cast<int>(rank) * HB;
        for (int kb = kb0; kb < kb1; ++kb) {
          if (!mbar_wait(&empty[stage], phase ^ 1u, ctx, 0x0701u)) { ok = false; break; }
          const uint32_t leader_full = mapa_shared(smem_u32(&full[stage]), 0);
          if (rank == 0) mbar_expect_tx(&full[stage], 2 * kStageBytes);  // both CTAs' bytes land here
          uint8_t* sa = smem + stage * kStageBytes;
          uint8_t* sb = sa + kOperandBytes;
          // one copy brings the three planes of a box: [plane][128 rows][64 k], or per 64-wide MN chunk [plane][64 k][64]
          if (A_KMAJOR) {
            tma_load_3d_pair(sa, &tmap_a, leader_full, kb * BK, m0, 0);
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) tma_load_3d_pair(sa + h * 24576, &tmap_a, leader_full, m0 + h * 64, kb * BK, 0);
          }
          if (B_KMAJOR) {
            tma_load_3d_pair(sb, &tmap_b, leader_full, kb * BK, n0, 0);
          } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) tma_load_3d_pair(sb + h * 24576, &tmap_b, leader_full, n0 + h * 64, kb * BK, 0);
          }
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      constexpr uint32_t idesc = idesc_bf16_f32(2 * BM, BN, !A_KMAJOR, !B_KMAJOR);
      // planes of A and B of the six partial products, smallest first
      constexpr int kPa[6] = {0, 2, 1, 0, 1, 0}, kPb[6] = {2, 0, 1, 1, 0, 0};
      int stage = 0;
      uint32_t phase = 0;
      int it = 0;
      bool ok = true;
      for (int item = pair; item < total && ok; item += npairs) {
        const int split = item / tiles;
        const int kb0 = static_cast<int>(static_cast<int64_t>(split) * p.num_kb / p.split_k);
        const int kb1 = static_cast<int>(static_cast<int64_t>(split + 1) * p.num_kb / p.split_k);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          const int buf = it & 1;
          if (!mbar_wait_cluster(&tmem_empty[buf], ((it >> 1) & 1u) ^ 1u, ctx, 0x0801u)) { ok = false; break; }
          if (!mbar_wait_cluster(&full[stage], phase, ctx, 0x0802u)) { ok = false; break; }
          tc_fence_after_sync();
          const uint32_t d_tmem = tmem_base + static_cast<uint32_t>(buf * BN);
          const uint32_t sa = smem_u32(smem + stage * kStageBytes);
          const uint32_t sb = sa + kOperandBytes;
#pragma unroll
          for (int t = 0; t < 6; ++t) {
#pragma unroll
            for (int k4 = 0; k4 < BK / 16; ++k4) {
              const uint64_t ad = A_KMAJOR ? smem_desc_sw128(sa + kPa[t] * 16384 + k4 * 32, 16, 1024)
                                           : smem_desc_sw128(sa + kPa[t] * 8192 + k4 * 2048, 24576, 1024);
              const uint64_t bd = B_KMAJOR ? smem_desc_sw128(sb + kPb[t] * 16384 + k4 * 32, 16, 1024)
                                           : smem_desc_sw128(sb + kPb[t] * 8192 + k4 * 2048, 24576, 1024);
              mma_bf16_ss_pair(d_tmem, ad, bd, idesc, (t > 0 || k4 > 0) ? 1u : 0u);
            }
          }
          mma_commit_pair(&empty[stage], 3);      // stage free in both CTAs once these MMAs have read it
          mma_commit_pair(&tmem_full[buf], 3);    // ... and the chain's sums are complete
          if (++stage == kStages) { stage = 0; phase ^= 1u; }
        }
      }
    }
  } else if (warp >= kFirstEpilogueWarp) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsEpilogue));
    const int quarter = warp & 3;                        // tensor-memory lanes [32 * quarter, +32)
    const int half = (warp - kFirstEpilogueWarp) >> 2;   // columns [128 * half, +128) of the tile
    uint8_t* strip = strips + (warp - kFirstEpilogueWarp) * kStripBytes;
    const uint32_t leader_empty0 = mapa_shared(smem_u32(&tmem_empty[0]), 0);
    const uint32_t leader_empty1 = mapa_shared(smem_u32(&tmem_empty[1]), 0);
    const uint64_t seed = p.ep.mode == PTJ_EPI_DROPOUT_RESID ? resolve_seed(p.ep.seed) : 0ull;
    int it = 0;
    bool ok = true;
    // the splitting pass's findings are read while the first tile is fetched and multiplied
    const int etid = threadIdx.x - kFirstEpilogueWarp * 32;
    int big = 0;
    for (int i = etid; i < p.num_flags; i += kEpilogueWarps * 32) big |= __ldcg(p.flags + i);
    if (big) atomicOr(epi_state, 1);
    epilogue_warps_sync();
    big = *epi_state & 1;  // the same in every block
    if (blockIdx.x == 0 && etid == 0) *p.any_flag = big;
    if (big) {  // let the issuing warps run through, unread, then multiply here
      for (int item = pair; item < total && ok; item += npairs) {
        const int split = item / tiles;
        const int nkb = static_cast<int>(static_cast<int64_t>(split + 1) * p.num_kb / p.split_k) -
                        static_cast<int>(static_cast<int64_t>(split) * p.num_kb / p.split_k);
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          ok = mbar_wait(&tmem_full[it & 1], (it >> 1) & 1u, ctx, 0x0901u);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          if (lane == 0) mbar_arrive_cluster((it & 1) == 0 ? leader_empty0 : leader_empty1);
        }
      }
      if (!ok) atomicOr(epi_state, 2);
      epilogue_warps_sync();  // (reached by every warp: the waits above are bounded)
      if (*epi_state == 1) product_by_fma<A_KMAJOR, B_KMAJOR>(p, reinterpret_cast<float*>(strips), seed, etid);
      ok = false;
    }
    for (int item = pair; item < total && ok; item += npairs) {
      const int split = item / tiles, tile = item - split * tiles;
      const int m_blk = tile % p.num_m, n_blk = tile / p.num_m;
      const int kb0 = static_cast<int>(static_cast<int64_t>(split) * p.num_kb / p.split_k);
      const int kb1 = static_cast<int>(static_cast<int64_t>(split + 1) * p.num_kb / p.split_k);
      uint64_t acc[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = 0ull;
#pragma unroll 1
      for (int kb = kb0; kb < kb1; ++kb, ++it) {
        const int buf = it & 1;
        ok = mbar_wait(&tmem_full[buf], (it >> 1) & 1u, ctx, 0x0901u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after_sync();
        const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + static_cast<uint32_t>(buf * BN + half * 128);
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          float r[32];
          tmem_ld_32x32f(taddr + c * 32, r);
          tmem_ld_wait();
#pragma unroll
          for (int j = 0; j < 16; ++j) acc[c * 16 + j] = f2_add(acc[c * 16 + j], f2_pack(r[2 * j], r[2 * j + 1]));
        }
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive_cluster(buf == 0 ? leader_empty0 : leader_empty1);
      }
      if (!ok) break;
      const int64_t row0 = static_cast<int64_t>(m_blk) * 2 * BM + static_cast<int64_t>(rank) * BM + quarter * 32;
      const int64_t row = row0 + lane;
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const int64_t n0 = static_cast<int64_t>(n_blk) * BN + half * 128 + c * 32;
        float v[32];
#pragma unroll
        for (int j = 0; j < 16; ++j) f2_unpack(f2_mul(acc[c * 16 + j], f2_pack(kUnscale, kUnscale)), v[2 * j], v[2 * j + 1]);
        if (p.split_k > 1) {
          float* w = p.workspace + static_cast<int64_t>(split) * p.M * p.N;
          if ((p.N & 3) == 0 && n0 + 32 <= p.N) {
            warp_store_block<float>(strip, w, p.N, row0, n0, p.M, v, lane);
          } else if (row < p.M) {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (n0 + j < p.N) w[row * p.N + n0 + j] = v[j];
          }
          continue;
        }
        const bool staged = p.ep.vec_ok && n0 + 32 <= p.N;  // warp-uniform
        const bool inside = epilogue_pre<float, 32>(p.ep, row, n0, v);
        float* out = static_cast<float*>(p.ep.c);
        float* aux_out = static_cast<float*>(p.ep.aux_out);
        if (p.ep.mode == PTJ_EPI_GELU && aux_out != nullptr) {
          if (staged) warp_store_block<float>(strip, aux_out, p.ep.ldc, row0, n0, p.M, v, lane);
          else if (inside) store_row<float, 32>(aux_out + row * p.ep.ldc, n0, p.N, false, v);
        }
        float side[32];
        if (const void* sptr = epilogue_side_input(p.ep)) {
          if (staged) warp_load_block<float>(strip, static_cast<const float*>(sptr), p.ep.ldc, row0, n0, p.M, side, lane);
          else if (inside) load_row<float, 32>(static_cast<const float*>(sptr) + row * p.ep.ldc, n0, p.N, false, side);
        }
        if (inside) epilogue_post<float, 32>(p.ep, row, n0, v, side, seed);
        if (staged) warp_store_block<float>(strip, out, p.ep.ldc, row0, n0, p.M, v, lane);
        else if (inside) store_row<float, 32>(out + row * p.ep.ldc, n0, p.N, false, v);
      }
    }
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    // give copies still in flight time to land before shared memory is handed back
    for (int i = 0; i < 64; ++i) __nanosleep(1000);
  }
  cluster_sync_all();  // neither CTA leaves (or frees tensor memory) while its peer may still signal it
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, 512);
  }
}

// Sum of the K parts (fixed order) followed by the full epilogue: one thread per row and group of eight columns.
__global__ void __launch_bounds__(256)
f32_finish_kernel(const float* __restrict__ ws, const int* __restrict__ any_flag, const EpilogueParams ep, int split_k) {
  grid_dep_sync();
  const int stored = *any_flag;  // the product kernel has stored the result itself
  const uint64_t seed = ep.mode == PTJ_EPI_DROPOUT_RESID ? resolve_seed(ep.seed) : 0ull;
  const int64_t groups = (ep.N + 7) / 8, total = ep.M * groups;
  const bool vec = (ep.N & 3) == 0;
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < total;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t m = i / groups, n0 = (i - m * groups) * 8;
    float acc[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[j] = 0.f;
    for (int k = 0; k < split_k; ++k) {
      const float* src = ws + (static_cast<int64_t>(k) * ep.M + m) * ep.N + n0;
      if (vec && n0 + 8 <= ep.N) {
        const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
        acc[0] += a.x; acc[1] += a.y; acc[2] += a.z; acc[3] += a.w;
        acc[4] += b.x; acc[5] += b.y; acc[6] += b.z; acc[7] += b.w;
      } else {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          if (n0 + j < ep.N) acc[j] += src[j];
      }
    }
    if (stored) return;
    epilogue_row_segment<float, 8>(ep, m, n0, acc, seed);
  }
}

// Which float32 products run here. A 256 x 256 tile costs the same however little of it is used and the splitting pass is
// a launch of its own, so 14 us is the least a product takes; the fused-multiply-add kernel (gemm.cu) is a serial walk
// along K: 7.4 us at K = 64, 12 us at K = 128, 20 us at K = 256, 36 us at K = 512 and 261 us at K = 4096 where its blocks
// all run at once, and 22-25 TFLOP/s where they do not. Measured (B200, device time, us, FMA -> here):
//   [512,128]x128: 12 -> 14   [512,1024]x128: 13 -> 16   [256,256]x256: 20 -> 19   [128,768]x768: 53 -> 19
//   [2048,768]x768: 114 -> 30   [4096,2304]x768: 592 -> 73   [4096,35376]x768: 9226 -> 928   [768,768]x4096: 317 -> 43
bool use_f32_tc(int64_t M, int64_t N, int64_t K) {
  if (M < 64 || N < 64 || K < 64) return false;
  return (K >= 256 && M * N >= (1LL << 13)) || M * N * K >= (1LL << 27);
}

// Parts of K: the product with the least of (rounds of the 74 pairs x K blocks of 3 072 clk) plus what writing and
// re-reading the parts costs (about 2.5 TB/s through the finishing kernel, and its launch).
int f32_split_k(int64_t M, int64_t N, int64_t K) {
  const int64_t tiles = ceil_div(M, 2 * BM) * ceil_div(N, BN), kb = ceil_div(K, BK);
  int best = 1;
  double best_us = 1e30;
  for (int s = 1; s <= 16 && s * 2 <= kb; ++s) {
    double us = static_cast<double>(ceil_div(tiles * s, kPairs)) * static_cast<double>(ceil_div(kb, s)) * 1.65;
    if (s > 1) us += 3.0 + static_cast<double>(s) * M * N * 8e-6 / 4.0;
    if (us < best_us * 0.97) {
      best_us = us;
      best = s;
    }
  }
  return best;
}

constexpr int kMaxSplitBlocks = kNumSMs * 16;
constexpr size_t kFlagBytes = (static_cast<size_t>(kMaxSplitBlocks + 1) * 4 + 255) / 256 * 256;

size_t plane_bytes(int64_t rows, int64_t cols) {  // multiple of 256
  return (static_cast<size_t>(3) * rows * ((cols + 7) / 8 * 8) * 2 + 255) / 256 * 256;
}

bool make_plane_map(CUtensorMap* t, const void* planes, int64_t rows, int64_t cols, bool kmajor) {
  const int64_t ldp = (cols + 7) / 8 * 8;
  const uint64_t dims[3] = {static_cast<uint64_t>(cols), static_cast<uint64_t>(rows), 3};
  const uint64_t str[2] = {static_cast<uint64_t>(ldp) * 2, static_cast<uint64_t>(rows) * ldp * 2};
  const uint32_t box[3] = {64, kmajor ? 128u : 64u, 3};
  return make_tmap_bf16(t, planes, 3, dims, str, box);
}

template <bool AK, bool BK_>
int launch_product(const CUtensorMap& ta, const CUtensorMap& tb, const F32Params& p, cudaStream_t st) {
  auto kern = gemm_f32_pair_kernel<AK, BK_>;
  static std::atomic<uint64_t> attr_done{0};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return PTJ_ERR_LAUNCH;
  if (!(attr_done.load(std::memory_order_acquire) & (1ull << dev))) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes) != cudaSuccess) {
      (void)cudaGetLastError();
      return PTJ_ERR_LAUNCH;
    }
    attr_done.fetch_or(1ull << dev, std::memory_order_release);
  }
  const int total = p.num_m * p.num_n * p.split_k;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(2 * (total < kPairs ? total : kPairs)));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = kSmemBytes;
  cfg.stream = st;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  if (cudaLaunchKernelEx(&cfg, kern, ta, tb, p) != cudaSuccess) {
    (void)cudaGetLastError();
    return PTJ_ERR_LAUNCH;
  }
  count_launch(1);
  return PTJ_OK;
}

}  // namespace

size_t gemm_f32_workspace_floats(int64_t M, int64_t N, int64_t K, bool a_kmajor, bool b_kmajor) {
  if (!use_f32_tc(M, N, K)) return 0;
  size_t bytes = plane_bytes(a_kmajor ? M : K, a_kmajor ? K : M) + plane_bytes(b_kmajor ? N : K, b_kmajor ? K : N);
  bytes += kFlagBytes;
  const int s = f32_split_k(M, N, K);
  if (s > 1) bytes += static_cast<size_t>(s) * M * N * 4;
  return bytes / 4;
}

int gemm_f32_tc(const float* a, const float* b, const EpilogueParams& ep, int64_t M, int64_t N, int64_t K, int64_t lda,
                int64_t ldb, bool a_kmajor, bool b_kmajor, float* workspace, cudaStream_t st) {
  uint8_t* ws = reinterpret_cast<uint8_t*>(workspace);
  const int64_t ar = a_kmajor ? M : K, ac = a_kmajor ? K : M, br = b_kmajor ? N : K, bc = b_kmajor ? K : N;
  SplitSrc sa{a, reinterpret_cast<__nv_bfloat16*>(ws), lda, ar, ac, (ac + 7) / 8 * 8};
  ws += plane_bytes(ar, ac);
  SplitSrc sb{b, reinterpret_cast<__nv_bfloat16*>(ws), ldb, br, bc, (bc + 7) / 8 * 8};
  ws += plane_bytes(br, bc);
  int* flags = reinterpret_cast<int*>(ws);
  ws += kFlagBytes;
  F32Params p{};
  p.ep = ep;
  p.M = M;
  p.N = N;
  p.num_m = static_cast<int>(ceil_div(M, 2 * BM));
  p.num_n = static_cast<int>(ceil_div(N, BN));
  p.num_kb = static_cast<int>(ceil_div(K, BK));
  p.split_k = f32_split_k(M, N, K);
  p.workspace = reinterpret_cast<float*>(ws);
  p.a = a;
  p.b = b;
  p.lda = lda;
  p.ldb = ldb;
  p.K = K;
  p.flags = flags;
  p.any_flag = flags + kMaxSplitBlocks;
  p.fault = fault_word();
  if (p.fault == nullptr) return PTJ_ERR_DEVICE;
  if (static_cast<int64_t>(p.num_m) * p.num_n * p.split_k > 0x3fffffffLL) return PTJ_ERR_BAD_SHAPE;
  CUtensorMap ta, tb;
  if (!make_plane_map(&ta, sa.dst, ar, ac, a_kmajor) || !make_plane_map(&tb, sb.dst, br, bc, b_kmajor)) return PTJ_ERR_LAUNCH;

  const int64_t groups = ar * (sa.ldp / 8) + br * (sb.ldp / 8);
  int64_t blocks = ceil_div(groups, 256);
  if (blocks > kMaxSplitBlocks) blocks = kMaxSplitBlocks;
  p.num_flags = static_cast<int>(blocks);
  launch_k(split_planes_kernel, static_cast<int>(blocks), 256, 0, st, sa, sb, flags);
  PTJ_CHECK_LAUNCH();
  const int rc = a_kmajor ? (b_kmajor ? launch_product<true, true>(ta, tb, p, st) : launch_product<true, false>(ta, tb, p, st))
                          : (b_kmajor ? launch_product<false, true>(ta, tb, p, st) : launch_product<false, false>(ta, tb, p, st));
  if (rc != PTJ_OK || p.split_k == 1) return rc;
  blocks = ceil_div(M * ceil_div(N, 8), 256);
  if (blocks > kNumSMs * 8) blocks = kNumSMs * 8;
  launch_k(f32_finish_kernel, static_cast<int>(blocks), 256, 0, st, p.workspace, p.any_flag, ep, p.split_k);
  PTJ_CHECK_LAUNCH();
  return PTJ_OK;
}

}  // namespace ptj

extern "C" size_t ptj_gemm_f32_workspace_floats(int64_t M, int64_t N, int64_t K, int a_kmajor, int b_kmajor) {
  if (M < 1 || N < 1 || K < 1 || M > (1LL << 30) || N > (1LL << 30) || K > (1LL << 30)) return 0;
  return ptj::gemm_f32_workspace_floats(M, N, K, a_kmajor != 0, b_kmajor != 0);
}
