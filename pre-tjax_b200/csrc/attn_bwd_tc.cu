// Causal flash attention backward on tcgen05 tensor cores (bf16 in, fp32 accumulate), heads up to 128 wide, any seq.
// Semantics: model_triton.py:801-811 / 550-577: with P = softmax(causal(Q K^T / sqrt(d))) recomputed from the saved row
// statistics and Pd = dropout(P):  dV = Pd^T dO,  dP = dO V^T,  dS = P o (dP o keep - delta) / sqrt(d) with
// delta = rowsum(dO o O),  dK = dS^T Q,  dQ = dS K.
//
// Three launches:
//   1. prep:   delta[q] and the log2-domain log-sum-exp of every query row
//   2. main:   persistent, warp-specialised block per SM. A work item is a (KV tile j, batch*head); its tiles are the
//              query tiles i >= j. dK_j and dV_j accumulate in tensor memory over the item; the product dS_ij K_j
//              (tile i's share of dQ_i) is written to an fp32 workspace.
//   3. reduce: dQ_i = sum over j <= i of the workspace tiles, in a fixed order, to bf16.
// No atomics on results, so every result is bit-reproducible (the reference adds dQ with tl.atomic_add, :938).
// PARTS: what probabilities and score gradients are multiplied as. 1: rounded to bf16. 3: split exactly into three bf16
// parts, three products each, so that the operands stay float32 (the sums run in the tensor cores' accumulators, which truncate
// where the general kernels round: of dK and dV 6e-4 to 1.1e-3 of the elements are not the float64 value rounded to bf16, there
// 2.3e-4 to 3.3e-4; their errors against float64 agree to four digits). There the operands that are summed over masked entries (Q, K, V,
// dO) pass through zero_nonfinite, and two more launches (the general kernels, which return at once unless an element
// was replaced or a result is not finite) put back what such an element reaches.
//
// Main kernel, 640 threads:
//   warp 0      one thread issues the TMA copies: K_j, V_j of an item, Q_i and dO_i of a tile
//   warp 1      issues S = Q_i K_j^T and dP = dO_i V_j^T (dP goes into the columns S occupied once the scores have
//               been read out)
//   warp 2      issues dV += Pd^T dO_i for every tile in stream order
//   warp 3      issues dK += dS^T Q_i in stream order, then the tile's dQ share dS K_j (one issuer per accumulator
//               keeps the accumulation order fixed)
//   warps 4..19 compute, in G groups that take the tiles of the block's stream in turn. Warp (quarter, c) of a group owns rows
//               32 quarter .. + 31 (tensor-memory lane = row) and the 32 G columns of block c of its tiles. Per tile, phase A
//               forms P and writes Pd to shared memory, phase B turns dP into dS in the same buffer. Two groups (PARTS = 1,
//               a buffer each): one group's exponentials overlap the other's loads, stores and barriers.
// Tensor memory (512 columns): S / dP, the dQ share, dV, dK; two of the first two each for heads up to 64.
// Masks are applied to packed pairs (two permutations and an AND for four elements) and the 1 / sqrt(d) of dS to the results:
// instruction issue and, per warp, the chain load - exponentials - store - barrier bound it. Measured, all launches, dropout
// 0.1: [8, 12, 1024, 64], flags given, 134 us (a thread per row of 128 columns, two groups of four warps: 154; 32 columns a
// thread, all warps on one tile: 143); flags drawn here 151 (177). [4, 12, 500, 64] 44 us (the float32 FMA kernels 282),
// [8, 12, 1024, 32] 188 (991), [8, 12, 1024, 128] 327 (3860).
#include "attn_tc_dev.cuh"

namespace ptj {
namespace {

using namespace attn_tc;

template <int DHP, int PARTS>
struct Cfg {
  static constexpr int kTB = T * DHP * 2;                              // one operand tile
  static constexpr int kG = PARTS == 1 ? 2 : 1;                        // groups of compute warps
  static constexpr int kNB = DHP == 64 ? 2 : 1;                        // S / dP and dQ-share buffers in tensor memory
  static constexpr int kWB = PARTS == 1 ? 2 : 1;                       // Pd / dS buffers, PARTS tiles each
  static constexpr int kKV = DHP == 64 ? 2 : 1;                        // item buffers: K then V
  static constexpr int kQG = DHP == 64 ? (PARTS == 1 ? 3 : 2) : 1;     // tile buffers: Q then dO
  static constexpr int kOffQG = kKV * 2 * kTB;
  static constexpr int kOffW = kOffQG + kQG * 2 * kTB;
  static constexpr int kOffBars = kOffW + kWB * PARTS * kPBytes;
  static constexpr int kNumBars = 3 * kKV + 3 * kQG + 6 * kNB + 4 * kWB + 2;
  static constexpr int kSmemBytes = kOffBars + kNumBars * 8 + 16 + 80 + 4 * 32 + 1024;  // (+ 32 last-tile entries)
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of a block");
  static constexpr uint32_t kColS = 0, kColDQ = kNB * T, kColDV = kColDQ + kNB * DHP, kColDK = kColDV + DHP;
  static_assert(kColDK + DHP <= 512, "tensor memory");
};
constexpr int kComputeWarps = 16;  // of all groups
constexpr int kThreads = 128 + 32 * kComputeWarps;
constexpr int kRegsIO = 56, kRegsCompute = 104;  // of the 96 a thread that 640 threads are launched with
constexpr int kTmemCols = 512;

struct Sched {
  int total, rounds, nq, BH;
  uint32_t bh_magic;  // ceil(2^32 / BH): x / BH == umulhi(x, bh_magic) for every x the kernel meets (checked on the host)
};

// Position in the stream of (item, query tile) pairs of one thread block; every role walks the same stream.
// Items are ordered heaviest first (KV tile 0 has the most query tiles) and dealt in boustrophedon order.
// last_tile (row_kstart): per round of this block, the last query tile whose rows reach into the item's KV tile (later
// query tiles mask all of its keys: they are skipped); nullptr = every item runs to the last query tile.
constexpr int kMaxRoundsTabled = 32;
struct Cursor {
  int n, ord, kt, bh, i, i1, g;
  bool valid;
  const int* last_tile;
  __device__ __forceinline__ void next_item(const Sched& s) {
    valid = false;
    while (++n < s.rounds) {
      const int pos = (n & 1) ? static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x);
      const int sp = n * static_cast<int>(gridDim.x) + pos;
      if (sp < s.total) {
        kt = s.BH == 1 ? sp : static_cast<int>(__umulhi(static_cast<uint32_t>(sp), s.bh_magic));  // sp / BH
        bh = sp - kt * s.BH;
        i = kt;
        i1 = last_tile != nullptr ? last_tile[n] : s.nq - 1;
        ++ord;
        valid = true;
        return;
      }
    }
  }
  __device__ __forceinline__ void init(const Sched& s, const int* last = nullptr) {
    n = -1; ord = -1; g = 0; kt = 0; bh = 0; i = 0; i1 = 0;
    last_tile = last;
    next_item(s);
  }
  __device__ __forceinline__ bool first(const Sched&) const { return i == kt; }
  __device__ __forceinline__ bool last(const Sched&) const { return i == i1; }
  __device__ __forceinline__ void advance(const Sched& s) {
    ++g;
    if (i == i1) next_item(s); else ++i;
  }
};

// ---- 1. per-row constants ------------------------------------------------------------------------------------------
// LANES (8 or 16) lanes per query row, eight elements each: delta = sum_d dO[q,d] O[q,d]; lse2 = (row_max + log(row_sum)) *
// log2(e). Clears the flag the main kernel raises.
template <int LANES>
__global__ void __launch_bounds__(256)
attn_bwd_prep_kernel(const RowView d_o, const RowView o_view, const float* __restrict__ row_max,
                     const float* __restrict__ row_sum, float* __restrict__ delta, float* __restrict__ lse2,
                     unsigned int* __restrict__ bad, int S, int H, int D, int64_t rows) {
  grid_dep_sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) *bad = 0u;
  const int64_t r = (static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x) / LANES;
  const int part = threadIdx.x % LANES;
  float acc = 0.f;
  if (r < rows && part * 8 < D) {
    const int64_t bh = r / S, q = r % S;
    const __nv_bfloat16* g = d_o.row(bh / H, bh % H, q) + part * 8;
    const __nv_bfloat16* o = o_view.row(bh / H, bh % H, q) + part * 8;
    float x[8], y[8];
    Elem<__nv_bfloat16>::load_vec(g, x);
    Elem<__nv_bfloat16>::load_vec(o, y);
#pragma unroll
    for (int i = 0; i < 8; ++i) acc = fmaf(x[i], y[i], acc);
  }
#pragma unroll
  for (int off = 1; off < LANES; off *= 2) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (r < rows && part == 0) {
    delta[r] = acc;
    lse2[r] = (row_max[r] + logf(row_sum[r])) * kLog2e;
  }
}

// ---- 3. dQ = sum of the per-KV-tile shares ---------------------------------------------------------------------------
// A share is stored as D / 4 blocks of four columns, 128 rows each (a warp of the main kernel writes 512 contiguous
// bytes per store): float4 index ((bh * ntri + qt (qt + 1) / 2 + kt) * D / 4 + c4) * 128 + row. One thread sums one
// float4 over kt; consecutive threads take consecutive rows.
__global__ void __launch_bounds__(256)
attn_dq_reduce_kernel(const float* __restrict__ part, const RowView dq, const int32_t* __restrict__ kstart,
                      unsigned int* __restrict__ bad, int S, int H, int nq, int D, float scale, int64_t total_vec) {
  grid_dep_sync();
  const int64_t v = static_cast<int64_t>(blockIdx.x) * 256 + threadIdx.x;
  if (v >= total_vec) return;
  const int d4 = D / 4;
  const int row = static_cast<int>(v % T);
  const int c4 = static_cast<int>((v / T) % d4);
  const int64_t tile_id = v / (T * d4);  // bh * nq + qt
  const int64_t bh = tile_id / nq;
  const int qt = static_cast<int>(tile_id % nq);
  const int64_t q = static_cast<int64_t>(qt) * T + row;
  if (q >= S) return;
  const int64_t ntri = static_cast<int64_t>(nq) * (nq + 1) / 2;
  const float4* src =
      reinterpret_cast<const float4*>(part) + ((bh * ntri + static_cast<int64_t>(qt) * (qt + 1) / 2) * d4 + c4) * T + row;
  float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
  // packed / padded batches: shares of KV tiles before the row's first key were either skipped by the main kernel (not
  // written) or are exact zeros; a row without keys sums nothing
  int kt0 = 0;
  if (kstart != nullptr) {
    const int k = __ldg(kstart + (bh / H) * S + q);
    kt0 = k > q ? qt + 1 : max(k, 0) / T;
  }
  for (int kt = kt0; kt <= qt; ++kt) {
    const float4 t = __ldcs(src + static_cast<int64_t>(kt) * T * d4);
    acc.x += t.x; acc.y += t.y; acc.z += t.z; acc.w += t.w;
  }
  acc.x *= scale; acc.y *= scale; acc.z *= scale; acc.w *= scale;  // the 1 / sqrt(d) of dS
  uint2 pk;
  pk.x = pack_bf16(acc.x, acc.y);
  pk.y = pack_bf16(acc.z, acc.w);
  *reinterpret_cast<uint2*>(dq.row(bh / H, bh % H, q) + c4 * 4) = pk;
  if (bad != nullptr && !(isfinite(acc.x) && isfinite(acc.y) && isfinite(acc.z) && isfinite(acc.w))) *bad = 1u;
}

// ---- 2. main kernel --------------------------------------------------------------------------------------------------
struct BwdViews {
  RowView dk, dv, k;
};

// bit l set: row `first + l` of K (l = this lane) holds an element that is not finite
__device__ __noinline__ uint32_t nonfinite_rows(const RowView& k, int b, int h, int first, int S, int D, int lane) {
  bool bad = false;
  if (first + lane < S) {
    const __nv_bfloat16* r = k.row(b, h, first + lane);
    for (int d = 0; d < D; ++d) bad = bad || !isfinite(__bfloat162float(r[d]));
  }
  return __ballot_sync(0xffffffffu, bad);
}

// MODE 0: no dropout mask; 1: Philox drawn in the kernel; 2: precomputed keep flags (p.keep_bits).
// p.kstart (optional): query row i attends keys [p.kstart[b, i], i] only (see the forward kernel); masked probabilities
// are exact zeros, and so is every product they enter.
template <int DHP, int PARTS, int MODE>
__global__ void __launch_bounds__(kThreads, 1)
attn_bwd_ws_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ CUtensorMap tm_g,
                   const float* __restrict__ delta, const float* __restrict__ lse2, float* __restrict__ dq_part,
                   unsigned int* __restrict__ bad, const __grid_constant__ BwdViews views, const AttnParams p,
                   const Sched sched) {
  using C = Cfg<DHP, PARTS>;
  constexpr int kTB = C::kTB, kNB = C::kNB, kWB = C::kWB, kKV = C::kKV, kQG = C::kQG;
  constexpr bool kExact = PARTS > 1;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = align1024(smem_raw);
  uint8_t* kv_s = sm;              // item buffer b: K at b * 2 tiles, V right behind it
  uint8_t* qg_s = sm + C::kOffQG;  // tile buffer x: Q at x * 2 tiles, dO right behind it
  uint8_t* w_s = sm + C::kOffW;
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + C::kOffBars);
  // completions of TMA copies and single MMA commits
  uint64_t* kv_full = bars;                // [kKV]
  uint64_t* qg_full = kv_full + kKV;       // [kQG]
  uint64_t* s_full = qg_full + kQG;        // [kNB]
  uint64_t* dp_full = s_full + kNB;        // [kNB]
  uint64_t* dq_full = dp_full + kNB;       // [kNB]
  uint64_t* dv_done = dq_full + kNB;       // [kWB] the dV MMA has read Pd
  uint64_t* dkq_done = dv_done + kWB;      // [kWB] the dK and dQ-share MMAs (one issuer, one commit) have read dS
  uint64_t* acc_full = dkq_done + kWB;     // the item's last dK MMA is done
  // two MMA commits each
  uint64_t* kv_empty = acc_full + 1;       // [kKV] last dP and last dQ share of the item
  uint64_t* qg_empty = kv_empty + kKV;     // [kQG] the tile's dV and dK MMAs are done (S, dP came before)
  // one arrival per compute warp of the tile's group
  uint64_t* s_free = qg_empty + kQG;       // [kNB] scores are in registers
  uint64_t* dp_free = s_free + kNB;        // [kNB] dP is in registers
  uint64_t* dq_free = dp_free + kNB;       // [kNB] the dQ share has been copied out
  uint64_t* pd_ready = dq_free + kNB;      // [kWB]
  uint64_t* ds_ready = pd_ready + kWB;     // [kWB]
  uint64_t* kv_ok = ds_ready + kWB;        // [kKV] K and V have no element left that is not finite (kExact)
  uint64_t* qg_ok = kv_ok + kKV;           // [kQG] the same of Q and dO
  uint64_t* acc_free = qg_ok + kQG;        // dV / dK have been copied out
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + C::kNumBars);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  volatile int* bad_s = abort_flag + 1;  // this block has met an element that is not finite
  uint32_t* rk_s = tmem_slot + 4;        // Philox round keys
  int* last_tab = reinterpret_cast<int*>(rk_s + 20);  // [kMaxRoundsTabled] last query tile of this block's items

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const AbortCtx ctx{abort_flag, p.fault};

  if (tid == 0) {
    for (uint64_t* b = bars; b < bars + C::kNumBars; ++b)
      mbar_init(b, b < kv_empty ? 1 : (b < s_free ? 2 : kComputeWarps / C::kG));
    *abort_flag = 0;
    *bad_s = 0;
    fence_barrier_init();
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
    prefetch_tensormap(&tm_g);
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, kTmemCols);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  grid_dep_sync();  // set-up above touches no global memory; everything below may
  const uint32_t tmem = *tmem_slot;
  if (MODE == 1) {  // the kernel draws its own keep flags: round keys of the (possibly device-resident) seed
    if (tid == 0) philox_round_keys(p.dr.seed, rk_s);
    __syncthreads();
  }
  // Query tiles none of whose rows reach into the item's KV tile are skipped. Warp w looks at the item of round w,
  // w + warps, ...: the last query tile with a row whose first key lies in or before the KV tile (the diagonal tile is
  // always visited).
  const int* last_tile = nullptr;
  if (p.kstart != nullptr && sched.rounds <= kMaxRoundsTabled) {
    for (int n = warp; n < sched.rounds; n += kThreads / 32) {
      const int pos = (n & 1) ? static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x);
      const int sp = n * static_cast<int>(gridDim.x) + pos;
      int last = 0;
      if (sp < sched.total) {
        const int kt = sp / sched.BH, bh = sp - kt * sched.BH;
        const int32_t* ks = p.kstart + static_cast<int64_t>(bh / p.H) * p.S;
        const int kv_end = kt * T + T;  // keys of the tile are < kv_end
        last = kt;
        for (int i = kt + 1; i < sched.nq; ++i) {
          bool reach = false;
          for (int r = lane; r < T && i * T + r < p.S; r += 32) {
            const int row = i * T + r, k = __ldg(ks + row);
            reach = reach || (k <= row && k < kv_end);  // the row has keys and its first one is in or before the tile
          }
          if (__any_sync(0xffffffffu, reach)) last = i;
        }
      }
      if (lane == 0) last_tab[n] = last;
    }
    __syncthreads();
    last_tile = last_tab;
  }
  constexpr uint32_t idesc_s = idesc_bf16_f32(T, T, false, false);   // Q K^T and dO V^T
  constexpr uint32_t idesc_t = idesc_bf16_f32(T, DHP, true, true);   // Pd^T dO and dS^T Q
  constexpr uint32_t idesc_q = idesc_bf16_f32(T, DHP, false, true);  // dS K

  // the copy / MMA warps hand registers to the compute warps (whole groups of four warps switch together)
  if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kRegsIO));

  // A polling role gives up when nothing has moved for the wait limit, or when another thread already aborted.
  auto stalled = [&](bool progress, long long& t_idle, unsigned int site) {
    if (progress) {
      t_idle = clock64();
      return false;
    }
    if (*abort_flag) return true;
    if (clock64() - t_idle > kWaitLimitCycles) {
      *abort_flag = 1;
      record_fault(p.fault, site);
      return true;
    }
    return false;
  };

  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    if (lane == 0) {
      Cursor ci, ct;  // items (K_j, V_j) and tiles (Q_i, dO_i) are two independent sequences
      ci.init(sched, last_tile);
      ct.init(sched, last_tile);
      long long t_idle = clock64();
      while (ci.valid || ct.valid) {
        bool progress = false;
        if (ci.valid) {
          const int b = ci.ord % kKV;
          if (mbar_try_wait(&kv_empty[b], ((ci.ord / kKV) & 1) ^ 1u)) {
            mbar_expect_tx(&kv_full[b], 2 * kTB);
            load_rows<DHP>(kv_s + b * 2 * kTB, &tm_k, &kv_full[b], ci.kt * T, ci.bh % p.H, ci.bh / p.H);
            load_rows<DHP>(kv_s + b * 2 * kTB + kTB, &tm_v, &kv_full[b], ci.kt * T, ci.bh % p.H, ci.bh / p.H);
            ci.next_item(sched);
            progress = true;
          }
        }
        if (ct.valid) {
          const int x = ct.g % kQG;
          if (mbar_try_wait(&qg_empty[x], ((ct.g / kQG) & 1) ^ 1u)) {
            mbar_expect_tx(&qg_full[x], 2 * kTB);
            load_rows<DHP>(qg_s + x * 2 * kTB, &tm_q, &qg_full[x], ct.i * T, ct.bh % p.H, ct.bh / p.H);
            load_rows<DHP>(qg_s + x * 2 * kTB + kTB, &tm_g, &qg_full[x], ct.i * T, ct.bh % p.H, ct.bh / p.H);
            ct.advance(sched);
            progress = true;
          }
        }
        if (stalled(progress, t_idle, 0x2101u)) break;
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer: S = Q K^T, then dP = dO V^T over it
    // (all lanes walk the streams so that addresses and descriptors stay warp-uniform; an elected lane issues)
    uint64_t* kv_in = kExact ? kv_ok : kv_full;
    uint64_t* qg_in = kExact ? qg_ok : qg_full;
    Cursor cs, cd;
    cs.init(sched, last_tile);
    cd.init(sched, last_tile);
    long long t_idle = clock64();
    while (cs.valid || cd.valid) {
      bool progress = false;
      if (cs.valid) {
        const int x = cs.g % kNB, st = cs.g % kQG;
        bool ready = mbar_try_wait(&qg_in[st], (cs.g / kQG) & 1) &&
                     mbar_try_wait(&dp_free[x], ((cs.g / kNB) & 1) ^ 1u);  // dP of tile g - kNB was read
        if (ready && cs.first(sched)) ready = mbar_try_wait(&kv_in[cs.ord % kKV], (cs.ord / kKV) & 1);
        if (__all_sync(0xffffffffu, ready)) {
          tc_fence_after_sync();
          const uint32_t qa = smem_u32(qg_s + st * 2 * kTB), ka = smem_u32(kv_s + (cs.ord % kKV) * 2 * kTB);
#pragma unroll
          for (int k16 = 0; k16 < DHP / 16; ++k16)
            mma_bf16_ss_elect(tmem + C::kColS + x * T, desc_kmajor(qa, k16), desc_kmajor(ka, k16), idesc_s, k16 > 0);
          mma_commit_elect(&s_full[x]);
          cs.advance(sched);
          progress = true;
        }
      }
      if (cd.valid && (!cs.valid || cd.g < cs.g)) {
        const int x = cd.g % kNB;
        if (__all_sync(0xffffffffu, mbar_try_wait(&s_free[x], (cd.g / kNB) & 1))) {
          tc_fence_after_sync();
          const uint32_t ga = smem_u32(qg_s + (cd.g % kQG) * 2 * kTB + kTB);
          const uint32_t va = smem_u32(kv_s + (cd.ord % kKV) * 2 * kTB + kTB);
#pragma unroll
          for (int k16 = 0; k16 < DHP / 16; ++k16)
            mma_bf16_ss_elect(tmem + C::kColS + x * T, desc_kmajor(ga, k16), desc_kmajor(va, k16), idesc_s, k16 > 0);
          mma_commit_elect(&dp_full[x]);
          if (cd.last(sched)) mma_commit_elect(&kv_empty[cd.ord % kKV]);
          cd.advance(sched);
          progress = true;
        }
      }
      if (__any_sync(0xffffffffu, stalled(progress, t_idle, 0x2201u))) break;
    }
  } else if (warp == 2) {
    // ---------------------------------------------------------------- MMA issuer: dV += Pd^T dO (stream order)
    Cursor c;
    c.init(sched, last_tile);
    bool ok = true;
    while (c.valid && ok) {
      const int x = c.g % kWB, st = c.g % kQG;
      bool w = mbar_wait(&pd_ready[x], (c.g / kWB) & 1, ctx, 0x2301u);
      if (w && c.first(sched)) w = mbar_wait(acc_free, (c.ord & 1) ^ 1u, ctx, 0x2302u);  // previous item copied out
      ok = __all_sync(0xffffffffu, w);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t wa = smem_u32(w_s + x * PARTS * kPBytes), ga = smem_u32(qg_s + st * 2 * kTB + kTB);
      const uint32_t acc = c.first(sched) ? 0u : 1u;
#pragma unroll
      for (int part = 0; part < PARTS; ++part)
#pragma unroll
        for (int k16 = 0; k16 < T / 16; ++k16)
          mma_bf16_ss_elect(tmem + C::kColDV, desc_rows_as_k(wa + part * kPBytes, k16), desc_rows_as_k(ga, k16), idesc_t,
                            part + k16 > 0 ? 1u : acc);
      mma_commit_elect(&dv_done[x]);
      mma_commit_elect(&qg_empty[st]);
      c.advance(sched);
    }
  } else if (warp == 3) {
    // ---------------------------------------------------------------- MMA issuer: dK += dS^T Q (stream order) and the
    // tile's dQ share dS K_j; both read dS, so one warp issues them back to back
    Cursor c;
    c.init(sched, last_tile);
    bool ok = true;
    while (c.valid && ok) {
      const int x = c.g % kWB, xq = c.g % kNB, st = c.g % kQG;
      bool w = mbar_wait(&ds_ready[x], (c.g / kWB) & 1, ctx, 0x2401u);
      // the first dK of an item overwrites the accumulator: the previous item must have been copied out (the dV
      // issuer waits for the same barrier)
      if (w && c.first(sched)) w = mbar_wait(acc_free, (c.ord & 1) ^ 1u, ctx, 0x2403u);
      ok = __all_sync(0xffffffffu, w);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t wa = smem_u32(w_s + x * PARTS * kPBytes), qa = smem_u32(qg_s + st * 2 * kTB);
      const uint32_t ka = smem_u32(kv_s + (c.ord % kKV) * 2 * kTB);
      const uint32_t acc = c.first(sched) ? 0u : 1u;
#pragma unroll
      for (int part = 0; part < PARTS; ++part)
#pragma unroll
        for (int k16 = 0; k16 < T / 16; ++k16)
          mma_bf16_ss_elect(tmem + C::kColDK, desc_rows_as_k(wa + part * kPBytes, k16), desc_rows_as_k(qa, k16), idesc_t,
                            part + k16 > 0 ? 1u : acc);
      mma_commit_elect(&qg_empty[st]);
      if (c.last(sched)) mma_commit_elect(acc_full);
      ok = __all_sync(0xffffffffu, mbar_wait(&dq_free[xq], ((c.g / kNB) & 1) ^ 1u, ctx, 0x2402u));  // share g - kNB copied out
      if (!ok) break;
      tc_fence_after_sync();
#pragma unroll
      for (int part = 0; part < PARTS; ++part)
#pragma unroll
        for (int k16 = 0; k16 < T / 16; ++k16)
          mma_bf16_ss_elect(tmem + C::kColDQ + xq * DHP, desc_kmajor(wa + part * kPBytes, k16), desc_rows_as_k(ka, k16), idesc_q,
                            part + k16 > 0 ? 1u : 0u);
      mma_commit_elect(&dq_full[xq]);
      mma_commit_elect(&dkq_done[x]);
      if (c.last(sched)) mma_commit_elect(&kv_empty[c.ord % kKV]);
      c.advance(sched);
    }
  } else if (warp >= 4) {
    // ---------------------------------------------------------------- compute warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kRegsCompute));
    constexpr int kGroupWarps = kComputeWarps / C::kG, kCW = 32 * C::kG, kWords = C::kG;
    const int quarter = warp & 3;                    // tensor-memory lane quarter this warp may read
    const int grp = (warp - 4) / kGroupWarps;
    const int cb = ((warp - 4) >> 2) % (4 / C::kG);  // its columns of a tile: kCW from kCW cb on
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t t_s = tmem + lane_base + C::kColS + cb * kCW;
    constexpr int kOut = DHP / 4 * C::kG;  // columns of a dQ share, of dV and of dK that this warp copies out
    const float f_keep = p.dr.train ? 1.f : p.dr.eval_scale;  // (1 wherever there is a mask)
    const uint32_t thr_hi = p.dr.thr16 << 16;
    const int ntri = p.nq * (p.nq + 1) / 2;
    const int d4 = p.D / 4;
    const uint64_t sc2 = pack2(p.scale_log2, p.scale_log2);

    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity, unsigned int site) {
      ok = __all_sync(0xffffffffu, mbar_wait(bar, parity & 1u, ctx, site));
      tc_fence_after_sync();
      return ok;
    };
    auto arrive = [&](uint64_t* bar) {
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(bar);
    };

    // this warp's share of the operands of one tile (and of its item, at the item's first tile)
    auto clean = [&](const Cursor& c) {
      auto sweep = [&](uint8_t* tiles) {
        bool any = false;
#pragma unroll
        for (int x = 0; x < 2 * kTB / kComputeWarps; x += 512)
          any = zero_nonfinite(tiles + (warp - 4) * (2 * kTB / kComputeWarps) + x + lane * 16) || any;
        if (any) {
          *bad_s = 1;
          *bad = 1u;
          __threadfence_block();
        }
        fence_proxy_async_smem();
      };
      if (c.first(sched)) {
        const int b = c.ord % kKV;
        if (!wait(&kv_full[b], c.ord / kKV, 0x2510u)) return;
        sweep(kv_s + b * 2 * kTB);
        arrive(&kv_ok[b]);
      }
      const int x = c.g % kQG;
      if (!wait(&qg_full[x], c.g / kQG, 0x2511u)) return;
      sweep(qg_s + x * 2 * kTB);
      arrive(&qg_ok[x]);
    };

    // copies the dQ share of tile g (its MMA is done or nearly so) to the workspace
    auto drain_dq = [&](int g, int64_t tile) {
      const int x = g % kNB;
      if (!wait(&dq_full[x], g / kNB, 0x2501u)) return;
      float4* dst = reinterpret_cast<float4*>(dq_part) + (tile * d4 + cb * (kOut / 4)) * T + row;  // [D / 4][128 rows]
#pragma unroll
      for (int x0 = 0; x0 < kOut; x0 += 16) {
        uint32_t t[16];
        tmem_ld_32x16(tmem + lane_base + C::kColDQ + x * DHP + cb * kOut + x0, t);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 4; ++i)
          if (cb * (kOut / 4) + x0 / 4 + i < d4)
            __stcs(dst + (x0 / 4 + i) * T, make_float4(__uint_as_float(t[4 * i]), __uint_as_float(t[4 * i + 1]),
                                                       __uint_as_float(t[4 * i + 2]), __uint_as_float(t[4 * i + 3])));
      }
      arrive(&dq_free[x]);
    };

    // What phase A leaves for phase B: P, float32 (kExact) or packed bf16 pairs; the keep flags; delta
    uint32_t kept[kExact ? kCW : kCW / 2];
    uint32_t keepw[kWords];
    float row_delta = 0.f;

    // Phase A: P = 2^(s c - lse), masked entries zero, to keep; dropout(P) to shared memory
    auto phase_a = [&](const Cursor& c) {
      const int x = c.g % kNB, xw = c.g % kWB;
      const int q_row = c.i * T + row;
      const bool real = q_row < p.S;
      const int64_t ri = static_cast<int64_t>(c.bh) * p.S + q_row;
      const float lse = real ? __ldg(lse2 + ri) : 0.f;
      row_delta = real ? __ldg(delta + ri) : 0.f;
      const int first_key = p.kstart != nullptr && real ? __ldg(p.kstart + static_cast<int64_t>(c.bh / p.H) * p.S + q_row) : 0;
      const int k0 = c.kt * T + cb * kCW;  // first key of this thread's columns
#pragma unroll
      for (int w = 0; w < kWords; ++w) {
        keepw[w] = 0xffffffffu;
        if (MODE == 1)
          keepw[w] = keep_word(rk_s, (static_cast<uint64_t>(c.bh) * p.S + q_row) * p.S + static_cast<uint64_t>(k0 + 32 * w),
                               p.dr.stream_id, thr_hi);
        if (MODE == 2)
          keepw[w] = __ldg(reinterpret_cast<const uint32_t*>(p.keep_bits) +
                           ((static_cast<int64_t>(c.bh) * ntri + c.i * (c.i + 1) / 2 + c.kt) * T + row) * 4 + cb * kWords + w);
      }
      if (!wait(&s_full[x], c.g / kNB, 0x2502u)) return;
      float s[kWords][32];
#pragma unroll
      for (int w = 0; w < kWords; ++w) tmem_ld_32x32f(t_s + x * T + 32 * w, s[w]);
      tmem_ld_wait();
      arrive(&s_free[x]);  // dP may now overwrite the scores
      const uint64_t nl2 = pack2(-lse, -lse);
      // (one answer for the warp: others may be raising the flag, and what follows is a warp's)
      const bool odd = kExact && __any_sync(0xffffffffu, *bad_s != 0);
      // keys after the row (diagonal tile), before its document, rows beyond the sequence
      const bool edge = c.i == c.kt || p.kstart != nullptr || c.i * T + T > p.S || odd;
      uint8_t* w_tile = w_s + xw * PARTS * kPBytes;
#pragma unroll
      for (int w = 0; w < kWords; ++w) {
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          float a, b;
          unpack2(fma2(pack2(s[w][i], s[w][i + 1]), sc2, nl2), a, b);
          s[w][i] = ex2_approx(a);
          s[w][i + 1] = ex2_approx(b);
        }
        if (edge) {
          uint32_t valid = real ? range_bits(first_key - k0 - 32 * w, q_row - k0 - 32 * w) : 0u;
          // a key with an element that is not finite (zeroed in the tile) has a true score of -inf in every row whose
          // statistics are finite; the other rows' results are not, whatever it contributes
          if (odd) valid &= ~nonfinite_rows(views.k, c.bh / p.H, c.bh % p.H, k0 + 32 * w, p.S, p.D, lane);
          if (__any_sync(0xffffffffu, valid != 0xffffffffu)) {
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (((valid >> i) & 1u) == 0u) s[w][i] = 0.f;
          }
        }
        if (w == 0 && !wait(&dkq_done[xw], (c.g / kWB) ^ 1, 0x2503u)) return;  // tile g - kWB's dS has been read
#pragma unroll
        for (int i8 = 0; i8 < 32; i8 += 8) {
          uint32_t pw[PARTS][4];
          if constexpr (kExact) {
#pragma unroll
            for (int i = i8; i < i8 + 8; ++i) kept[32 * w + i] = __float_as_uint(s[w][i]);
          }
          if (MODE == 0 && f_keep != 1.f) {  // evaluation
            float t[8];
            uint32_t pu[1][4];
            if constexpr (!kExact) {
              split8<1>(s[w] + i8, pu);
#pragma unroll
              for (int i = 0; i < 4; ++i) kept[16 * w + i8 / 2 + i] = pu[0][i];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) t[i] = s[w][i8 + i] * f_keep;
            split8<PARTS>(t, pw);
          } else {
            split8<PARTS>(s[w] + i8, pw);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if constexpr (!kExact) kept[16 * w + i8 / 2 + i] = pw[0][i];
              if (MODE != 0) {
                const uint32_t m = pair_mask(keepw[w], i8 / 2 + i);
#pragma unroll
                for (int part = 0; part < PARTS; ++part) pw[part][i] &= m;
              }
            }
          }
          store8<PARTS>(w_tile, row, (cb * kCW + 32 * w + i8) >> 3, pw);
        }
      }
      fence_proxy_async_smem();
      arrive(&pd_ready[xw]);
    };

    // Phase B: sqrt(d) dS = P o (dP o keep - delta) into the same buffer, once the dV MMA has read Pd (dK and dQ take the
    // factor 1 / sqrt(d) when they are stored)
    auto phase_b = [&](const Cursor& c) {
      const int x = c.g % kNB, xw = c.g % kWB;
      if (!wait(&dp_full[x], c.g / kNB, 0x2504u)) return;
      uint8_t* w_tile = w_s + xw * PARTS * kPBytes;
      const uint64_t nd2 = pack2(-row_delta, -row_delta), fk2 = pack2(f_keep, f_keep);
      const bool odd = kExact && __any_sync(0xffffffffu, !isfinite(row_delta));
#pragma unroll
      for (int w = 0; w < kWords; ++w) {
        float s[32];
        tmem_ld_32x32f(t_s + x * T + 32 * w, s);
        tmem_ld_wait();
        if (w == kWords - 1) arrive(&dp_free[x]);  // the scores of tile g + kNB may now overwrite dP
#pragma unroll
        for (int i = 0; i < 32; i += 2) {
          uint64_t pr;
          if constexpr (kExact) pr = pack2(__uint_as_float(kept[32 * w + i]), __uint_as_float(kept[32 * w + i + 1]));
          else pr = pack2(bf16_lo(kept[16 * w + i / 2]), bf16_hi(kept[16 * w + i / 2]));
          uint64_t d;
          if (MODE != 0) d = add2(pack2(masked(s[i], keepw[w], i), masked(s[i + 1], keepw[w], i + 1)), nd2);
          else d = fma2(pack2(s[i], s[i + 1]), fk2, nd2);
          unpack2(mul2(pr, d), s[i], s[i + 1]);
        }
        if constexpr (kExact) {
          if (odd) {  // masked entries stay zeros in a row whose O or dO is not finite
#pragma unroll
            for (int i = 0; i < 32; ++i)
              if (kept[32 * w + i] == 0u) s[i] = 0.f;
          }
        }
        if (w == 0 && !wait(&dv_done[xw], c.g / kWB, 0x2505u)) return;
#pragma unroll
        for (int i8 = 0; i8 < 32; i8 += 8) {
          uint32_t pw[PARTS][4];
          split8<PARTS>(s + i8, pw);
          store8<PARTS>(w_tile, row, (cb * kCW + 32 * w + i8) >> 3, pw);
        }
      }
      fence_proxy_async_smem();
      arrive(&ds_ready[xw]);
    };

    // the item ends with this tile: its dV and dK rows
    auto copy_out = [&](const Cursor& c) {
      const int kv_row = c.kt * T + row;
      bool odd = false;
#pragma unroll
      for (int which = 0; which < 2; ++which) {  // dV is complete (phase B waited for it) while the last dK MMA still runs
        if (which == 1 && !wait(acc_full, c.ord, 0x2506u)) return;
        const float mul = which == 0 ? 1.f : p.scale;
        const RowView& view = which == 0 ? views.dv : views.dk;
        __nv_bfloat16* dst = view.row(c.bh / p.H, c.bh % p.H, kv_row);
#pragma unroll
        for (int x0 = 0; x0 < kOut; x0 += 16) {
          const int col = cb * kOut + x0;
          uint32_t t[16];
          tmem_ld_32x16(tmem + lane_base + (which == 0 ? C::kColDV : C::kColDK) + col, t);
          tmem_ld_wait();
#pragma unroll
          for (int c8 = 0; c8 < 2; ++c8) {
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              v[i] = __uint_as_float(t[c8 * 8 + i]) * mul;
              if (kExact) odd = odd || !isfinite(v[i]);
            }
            if (kv_row < p.S && col + c8 * 8 < p.D) Elem<__nv_bfloat16>::store_vec(dst + col + c8 * 8, v);
          }
        }
      }
      if (kExact && odd) *bad = 1u;
      arrive(acc_free);
    };

    Cursor c;
    c.init(sched, last_tile);
    int64_t share = -1;  // workspace tile of the dQ share still in tensor memory
    int share_g = 0;
    if (kExact && c.valid) clean(c);
    while (c.valid && ok) {
      if (C::kG > 1 && c.g % C::kG != grp) {
        c.advance(sched);
        continue;
      }
      phase_a(c);
      if (!ok) break;
      if (share >= 0) drain_dq(share_g, share);
      if (!ok) break;
      if (kExact && kQG > 1) {  // the next tile's operands have been in shared memory since tile g - 1 was done
        Cursor n = c;
        n.advance(sched);
        if (n.valid) clean(n);
        if (!ok) break;
      }
      phase_b(c);
      if (!ok) break;
      share = static_cast<int64_t>(c.bh) * ntri + c.i * (c.i + 1) / 2 + c.kt;
      share_g = c.g;
      if (c.last(sched)) copy_out(c);
      if (!ok) break;
      c.advance(sched);
      if (kExact && kQG == 1 && c.valid) clean(c);  // its buffer was only free once tile g was done
    }
    if (ok && share >= 0) drain_dq(share_g, share);
  }

  __syncwarp();
  tc_fence_before_sync();
  __syncthreads();
  if (*abort_flag) {
    for (int i = 0; i < 64; ++i) __nanosleep(1000);  // let copies in flight land before shared memory is released
    __syncthreads();
  }
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem, kTmemCols);
  }
}

struct BwdLaunch {
  CUtensorMap tq, tk, tv, tg;
  float *part, *delta, *lse2;
  unsigned int* bad;
  BwdViews views;
  AttnParams p;
  int mode;
};
template <int DHP, int PARTS>
int launch_bwd(const BwdLaunch& l, cudaStream_t st) {
  using C = Cfg<DHP, PARTS>;
  using Kern = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const CUtensorMap, const float*,
                        const float*, float*, unsigned int*, const BwdViews, const AttnParams, const Sched);
  static const Kern kerns[3] = {attn_bwd_ws_kernel<DHP, PARTS, 0>, attn_bwd_ws_kernel<DHP, PARTS, 1>,
                                attn_bwd_ws_kernel<DHP, PARTS, 2>};
  const Kern kern = kerns[l.mode];
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) {
    (void)cudaGetLastError();
    return PTJ_ERR_LAUNCH;
  }
  Sched s;
  s.nq = l.p.nq;
  s.BH = l.p.BH;
  s.total = l.p.nq * l.p.BH;
  const int grid = s.total < kNumSMs ? s.total : kNumSMs;
  s.rounds = (s.total + grid - 1) / grid;
  s.bh_magic = static_cast<uint32_t>(((1ull << 32) + s.BH - 1) / s.BH);
  launch_k(kern, grid, kThreads, C::kSmemBytes, st, l.tq, l.tk, l.tv, l.tg, l.delta, l.lse2, l.part, l.bad, l.views, l.p, s);
  PTJ_CHECK_LAUNCH();
  return PTJ_OK;
}

}  // namespace

bool attn_tc_supported(const ptj_attn_shape& sh, const void* const* ptrs, int nptrs) {
  if (sh.d_head < 16 || sh.d_head > 128 || sh.d_head % 8 != 0 || sh.seq > (1 << 20)) return false;
  const int64_t bh = sh.batch * sh.heads, items = bh * ceil_div(sh.seq, T);
  if (items * bh >= (1LL << 32)) return false;  // exactness bound of the kernels' reciprocal division by bh
  for (int i = 0; i < nptrs; ++i)
    if (!aligned16(ptrs[i])) return false;
  const int64_t* sts[4] = {sh.q_strides, sh.k_strides, sh.v_strides, sh.o_strides};
  for (const int64_t* st : sts) {
    if (st[0] % 8 != 0 || st[1] % 8 != 0 || st[2] % 8 != 0) return false;
    if ((sh.batch > 1 && st[0] <= 0) || (sh.heads > 1 && st[1] <= 0) || (sh.seq > 1 && st[2] < sh.d_head)) return false;
  }
  return ptj_device_check() == PTJ_OK;
}

size_t attn_bwd_tc_workspace_bytes(const ptj_attn_shape& sh) {
  const int64_t nq = ceil_div(sh.seq, T), bh = sh.batch * sh.heads;
  const int64_t part = bh * (nq * (nq + 1) / 2) * T * sh.d_head;  // dQ shares
  const int64_t rows = bh * sh.seq;                               // delta, lse2
  return static_cast<size_t>(part + 2 * rows + 4) * sizeof(float);  // (+ the flag)
}

int attn_bwd_tc(const void* d_o, const void* q, const void* k, const void* v, const void* o, const float* row_max,
                const float* row_sum, void* dq, void* dk, void* dv, const ptj_attn_shape& sh,
                const ptj_attn_shape& dsh, const AttnDropout& dr, const uint32_t* keep_bits,
                const int32_t* row_kstart, void* workspace, size_t workspace_bytes, cudaStream_t st) {
  if (workspace == nullptr || workspace_bytes < attn_bwd_tc_workspace_bytes(sh) || !aligned16(workspace))
    return PTJ_ERR_WORKSPACE;
  BwdLaunch l;
  if (!make_map(&l.tq, q, sh, sh.q_strides) || !make_map(&l.tk, k, sh, sh.k_strides) ||
      !make_map(&l.tv, v, sh, sh.v_strides) || !make_map(&l.tg, d_o, sh, sh.o_strides))
    return PTJ_ERR_LAUNCH;
  l.p = make_params(sh, dr);
  const AttnParams& p = l.p;
  if (p.fault == nullptr) return PTJ_ERR_DEVICE;
  l.p.keep_bits = reinterpret_cast<const uint4*>(keep_bits);
  l.p.kstart = row_kstart;
  const bool masked = dr.train && dr.thr16 != 0u;
  l.mode = !masked ? 0 : (p.keep_bits != nullptr ? 2 : 1);
  const int64_t rows = static_cast<int64_t>(p.BH) * p.S;
  l.part = static_cast<float*>(workspace);
  l.delta = l.part + static_cast<int64_t>(p.BH) * (p.nq * (p.nq + 1) / 2) * T * p.D;
  l.lse2 = l.delta + rows;
  l.bad = reinterpret_cast<unsigned int*>(l.lse2 + rows);
  l.views = BwdViews{make_view(dk, dsh.k_strides), make_view(dv, dsh.v_strides), make_view(k, sh.k_strides)};
  const RowView g_view = make_view(d_o, sh.o_strides), o_view = make_view(o, sh.o_strides);
  if (p.D <= 64)
    launch_k(attn_bwd_prep_kernel<8>, static_cast<unsigned>((rows * 8 + 255) / 256), 256, 0, st, g_view, o_view, row_max, row_sum,
             l.delta, l.lse2, l.bad, p.S, p.H, p.D, rows);
  else
    launch_k(attn_bwd_prep_kernel<16>, static_cast<unsigned>((rows * 16 + 255) / 256), 256, 0, st, g_view, o_view, row_max, row_sum,
             l.delta, l.lse2, l.bad, p.S, p.H, p.D, rows);
  PTJ_CHECK_LAUNCH();
  const bool exact = !attn_bf16_probabilities(sh);
  const int rc = p.D > 64 ? launch_bwd<128, 3>(l, st) : (exact ? launch_bwd<64, 3>(l, st) : launch_bwd<64, 1>(l, st));
  if (rc != PTJ_OK) return rc;
  const int64_t total_vec = static_cast<int64_t>(p.BH) * p.nq * T * (p.D / 4);
  launch_k(attn_dq_reduce_kernel, static_cast<unsigned>((total_vec + 255) / 256), 256, 0, st, l.part, make_view(dq, dsh.q_strides),
           row_kstart, exact ? l.bad : nullptr, p.S, p.H, p.nq, p.D, p.scale, total_vec);
  PTJ_CHECK_LAUNCH();
  if (!exact) return PTJ_OK;
  return attn_bwd_simt(d_o, q, k, v, o, row_max, row_sum, dq, dk, dv, row_kstart, sh, dsh, dr, PTJ_BF16, l.bad, st);
}

}  // namespace ptj
