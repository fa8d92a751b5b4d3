// Causal flash attention forward on tcgen05 tensor cores (bf16 in, fp32 accumulate), heads up to 128 wide, any seq, float32
// probabilities. (attn_fwd_tc64.cu: whole tiles of 64-wide heads, whose probabilities are rounded to bf16.)
// Semantics: model_triton.py:608-611 / 510-517: softmax of the causally masked scaled scores, dropout on the
// probabilities (no rescale), times V; the row maximum and row sum of exponentials are saved (acts0 / acts1, :699-700).
//
// Persistent, warp-specialised thread block (one per SM; 16 softmax warps for heads up to 64, 8 beyond):
//   warp 0      one thread issues the TMA copies: Q of a work item, K tiles, V tiles, as independent sequences
//   warp 1      issues the score MMAs S = Q K^T, up to two tiles ahead of the softmax
//   warp 2      issues the output MMAs O_x += P[:, block c] V[block c, :] for the NC column blocks of a tile
//   warps 4..   softmax, in G groups that take the tiles of the block's stream in turn, so that one group's exponentials
//               overlap the other's loads, stores and barriers. Warp (quarter, c) of a group owns rows 32 quarter .. + 31
//               (tensor-memory lane = row, one row per thread) and the 128 / NC columns of block c of the group's tiles. Every
//               (group, block) has its own reference exponent, row sums and output accumulator, so the warps of a row never
//               meet before the item ends; then the group that got the last tile merges the G NC states of each row
//               (log-sum-exp merge in a fixed order) and writes it.
// A probability is split exactly into three bf16 parts, three products each; the operands of S are bf16 as they are. Sums run in
// the tensor cores' float32 accumulators, which truncate at every step: S over a head, O over a row's whole length. Errors
// against float64 beside those of the float32 FMA kernels, [4, 12, 500, 64] and [2, 16, 1024, 128]: row maximum 7.0e-8 (3.8e-8) and
// 1.5e-7 (5.5e-8), row sum 1.4e-7 (1.1e-7) and 2.6e-7 (1.7e-7); O, rounded to bf16, 1.592912e-3 and 1.607495e-3 on both.
// Work items = (query tile, batch*head), heaviest first, dealt to the blocks in boustrophedon order; all tiles of a
// block's items form one stream, so the next item's first tiles overlap the tail of the current one.
// Tensor memory: two S buffers at columns [0,256), the G NC accumulators at [256,512).
// Bound by the latencies a softmax warp meets in a row on its tile (tensor-memory loads, barriers, exponentials), not by a
// pipe. Measured, dropout 0.1, flags drawn here: [4, 12, 500, 64] 22 us (the float32 FMA kernels 95), [8, 12, 1024, 32] 111
// (338), [8, 12, 1024, 128] 136 (837). (With one bf16 part, [8, 12, 1024, 64]: 41.8 us with flags given, 74.6 with flags drawn
// here, against 40.8 and 69 of attn_fwd_tc64.cu; all 16 warps on one tile, 32 columns a thread: 65.)
#include "attn_fwd_sched.cuh"

namespace ptj {
namespace {

using namespace attn_tc;

constexpr int kParts = 3;  // bf16 parts of a probability

template <int DHP>
struct Cfg {
  static constexpr int kG = DHP == 64 ? 2 : 1;     // groups
  static constexpr int kNC = 2;                    // column blocks of a tile
  static constexpr int kCW = T / kNC;              // columns of a block
  static constexpr int kGroupWarps = 4 * kNC;
  static constexpr int kWarps = kG * kGroupWarps;  // softmax warps
  static constexpr int kAcc = kG * kNC;            // accumulators
  static constexpr int kThreads = 128 + 32 * kWarps;
  static constexpr int kTB = T * DHP * 2;          // one operand tile
  // shared memory, in tiles: what fits beside the probabilities
  static constexpr int kQ = DHP == 64 ? 2 : 1;
  static constexpr int kK = DHP == 64 ? 2 : 1;
  static constexpr int kV = DHP == 64 ? 3 : 1;
  static constexpr int kOffK = kQ * kTB;
  static constexpr int kOffV = kOffK + kK * kTB;
  static constexpr int kOffP = kOffV + kV * kTB;
  static constexpr int kOffStats = kOffP + kParts * kPBytes;  // float [kAcc][3][128]
  static constexpr int kOffBars = kOffStats + kAcc * 3 * T * 4;
  static constexpr int kNumBars = 2 * (kQ + kK + kV) + 4 + kG + 1 + 2;
  static constexpr int kSmemBytes = kOffBars + kNumBars * 8 + 16 + 80 + 4 * 32 + 1024;  // (+ 32 first-tile entries)
  static_assert(kSmemBytes <= 227 * 1024, "shared memory of a block");
  // of 96 (640 threads) or 168 (384 threads) a thread at launch
  static constexpr int kRegsIO = DHP == 64 ? 56 : 40, kRegsSoftmax = DHP == 64 ? 104 : 232;
};
constexpr int kSBufs = 2;
constexpr int kTmemCols = 512;
constexpr uint32_t kColO = kSBufs * T;

// An item one of whose V tiles held an infinity or a NaN (replaced by zero before it was multiplied): the products of a
// row's attended probabilities with those elements, columns [col0, col0 + 16), added to o. A whole warp, a row a lane (`live`:
// the row exists and attends keys). Each lane looks at one key's elements, so that keys without such elements cost a
// thirty-second of a load; a key's probabilities are formed where they may change something: a column that is NaN stays NaN,
// and with all of them the rest of the keys is left out. Forward passes of
// [8, 12, 1024, 32] (117 us) and [8, 12, 1024, 128] (140) with one NaN in V: 138 and 199 us (a thread for itself, key by key, and
// in all later items of the block: 4751 and 8352), with nothing else in V: 220 and 391 (24 and 246 ms).
__device__ __noinline__ void add_nonfinite_v(float (&o)[16], const RowView& q, const RowView& k, const RowView& v, const AttnParams& p,
                                             const uint32_t* rk_s, int mode, int bh, int q_row, int first_key, bool live, int col0,
                                             float m_true) {
  const int b = bh / p.H, h = bh % p.H, lane = threadIdx.x & 31;
  const int vecs = min(2, (p.D - col0) / 8);
  if (vecs <= 0) return;
  const uint32_t all = (1u << (8 * vecs)) - 1u;
  const int begin = __reduce_min_sync(0xffffffffu, live ? max(first_key, 0) : 0x7fffffff);
  const int end = __reduce_max_sync(0xffffffffu, live ? q_row : -1);
  uint32_t nan = 0u;  // columns of this lane's row that are NaN by now
  for (int j0 = begin; j0 <= end; j0 += 32) {
    uint32_t bad = 0u;
    if (j0 + lane <= end) {
      const uint4* vr = reinterpret_cast<const uint4*>(v.row(b, h, j0 + lane) + col0);
      for (int x = 0; x < vecs; ++x) {
        const uint4 e = vr[x];
        const uint32_t w[4] = {e.x, e.y, e.z, e.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          if ((w[i] & 0x7f80u) == 0x7f80u) bad |= 1u << (8 * x + 2 * i);
          if ((w[i] & 0x7f800000u) == 0x7f800000u) bad |= 2u << (8 * x + 2 * i);
        }
      }
    }
    for (uint32_t keys = __ballot_sync(0xffffffffu, bad != 0u); keys != 0u; keys &= keys - 1u) {
      const int src = __ffs(keys) - 1, j = j0 + src;
      const uint32_t cols = __shfl_sync(0xffffffffu, bad, src);
      if (!live || j < first_key || j > q_row || (cols & ~nan) == 0u) continue;  // (each lane goes its own way to the next key)
      const uint4 *qr = reinterpret_cast<const uint4*>(q.row(b, h, q_row)), *kr = reinterpret_cast<const uint4*>(k.row(b, h, j));
      float s = 0.f;
      for (int d = 0; d < p.D / 8; ++d) {
        const uint4 x = qr[d], y = kr[d];
        const uint32_t xw[4] = {x.x, x.y, x.z, x.w}, yw[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) s = fmaf(bf16_hi(xw[i]), bf16_hi(yw[i]), fmaf(bf16_lo(xw[i]), bf16_lo(yw[i]), s));
      }
      float w = ex2_approx((s - m_true) * p.scale_log2);
      if (mode != 0) {
        const uint64_t idx = (static_cast<uint64_t>(bh) * p.S + q_row) * p.S + j;
        uint32_t keep;
        if (mode == 1) {
          keep = keep_word(rk_s, idx, p.dr.stream_id, p.dr.thr16 << 16) & 1u;
        } else {
          const int qt = q_row / T, kt = j / T;
          const uint32_t* words = reinterpret_cast<const uint32_t*>(p.keep_bits);
          const int64_t tile = static_cast<int64_t>(bh) * (p.nq * (p.nq + 1) / 2) + qt * (qt + 1) / 2 + kt;
          keep = (__ldg(words + (tile * T + q_row % T) * 4 + (j % T) / 32) >> (j & 31)) & 1u;
        }
        if (keep == 0u) w = 0.f;
      }
      const __nv_bfloat16* vr = v.row(b, h, j) + col0;
#pragma unroll
      for (int i = 0; i < 16; ++i)
        if ((cols >> i) & 1u) {
          o[i] += w * __bfloat162float(vr[i]);
          if (isnan(o[i])) nan |= 1u << i;
        }
    }
    if (__all_sync(0xffffffffu, !live || nan == all)) break;
  }
}

struct FwdViews {
  RowView q, k, v, o;
};

// MODE 0: no dropout mask; 1: Philox drawn in the kernel; 2: precomputed keep flags (p.keep_bits).
// p.kstart (optional): query row i attends keys [p.kstart[b, i], i] only (packed documents / padding, the block-diagonal x
// causal x padding masks of the reference's collator, tokenized_dataset.py:110-131); a row whose range is empty gets a
// zero output row and the statistics (row_max, row_sum) = (0, 1).
template <int DHP, int MODE>
__global__ void __launch_bounds__(Cfg<DHP>::kThreads, 1)
attn_fwd_ws_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
                   const __grid_constant__ CUtensorMap tm_v, const __grid_constant__ FwdViews views,
                   float* __restrict__ row_max, float* __restrict__ row_sum, const __grid_constant__ AttnParams p,
                   const Sched sched) {
  using C = Cfg<DHP>;
  constexpr int kTB = C::kTB;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* sm = align1024(smem_raw);
  uint8_t* q_s = sm;
  uint8_t* k_s = sm + C::kOffK;
  uint8_t* v_s = sm + C::kOffV;
  uint8_t* p_s = sm + C::kOffP;
  float* stats = reinterpret_cast<float*>(sm + C::kOffStats);
  uint64_t* bars = reinterpret_cast<uint64_t*>(sm + C::kOffBars);
  uint64_t* q_full = bars;                  // [kQ]
  uint64_t* q_empty = q_full + C::kQ;
  uint64_t* k_full = q_empty + C::kQ;       // [kK]
  uint64_t* k_empty = k_full + C::kK;
  uint64_t* v_full = k_empty + C::kK;       // [kV]
  uint64_t* v_empty = v_full + C::kV;
  uint64_t* s_full = v_empty + C::kV;       // [2]
  uint64_t* o_full = s_full + kSBufs;       // [kG] per group: its tile's output MMAs, and all before, are done
  uint64_t* s_free = o_full + C::kG;        // [2] one arrival per warp of the tile's group from here on
  uint64_t* p_ready = s_free + kSBufs;
  uint64_t* stats_full = p_ready + 1;   // the item's row states are in shared memory (all softmax warps)
  uint64_t* o_free = stats_full + 1;        // the item's accumulators and states have been read
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(o_free + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  // [2] ordinal + 1 of the last even / odd item of which a V tile held an element that is not finite. (An item's slot is
  // written again two items on, and that one's tiles wait for this one's rows to be merged.)
  volatile int* bad_v = abort_flag + 1;
  uint32_t* rk_s = tmem_slot + 4;        // Philox round keys (MODE 1)
  int* first_tab = reinterpret_cast<int*>(rk_s + 20);  // [kMaxRoundsTabled] first KV tile of this block's items

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const AbortCtx ctx{abort_flag, p.fault};

  if (tid == 0) {
    for (uint64_t* b = bars; b < s_free; ++b) mbar_init(b, 1);  // TMA / MMA completions
    for (uint64_t* b = s_free; b < o_free + 1; ++b) mbar_init(b, b == stats_full ? C::kWarps : C::kGroupWarps);
    *abort_flag = 0;
    bad_v[0] = bad_v[1] = 0;
    fence_barrier_init();
    prefetch_tensormap(&tm_q);
    prefetch_tensormap(&tm_k);
    prefetch_tensormap(&tm_v);
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
  // Whole KV tiles before the first key of every row of a query tile are skipped. Warp w looks at the item of round
  // w, w + warps, ...: the smallest first key over the tile's rows that have keys at all (none: only the diagonal
  // tile is visited, it masks everything).
  const int* first_tile = nullptr;
  if (p.kstart != nullptr && sched.rounds <= kMaxRoundsTabled) {
    for (int n = warp; n < sched.rounds; n += C::kThreads / 32) {
      const int pos = (n & 1) ? static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x);
      const int sp = n * static_cast<int>(gridDim.x) + pos;
      int first = 0;
      if (sp < sched.total) {
        const int t = sp / sched.BH;
        const int qt = sched.nq - 1 - t, bh = sp - t * sched.BH;
        const int32_t* ks = p.kstart + static_cast<int64_t>(bh / p.H) * p.S + static_cast<int64_t>(qt) * T;
        int lo = 0x7fffffff;
        for (int r = lane; r < T && qt * T + r < p.S; r += 32) {
          const int k = __ldg(ks + r);
          if (k <= qt * T + r) lo = min(lo, k);  // (k > row: the row has no keys)
        }
        lo = __reduce_min_sync(0xffffffffu, lo);
        first = lo == 0x7fffffff ? qt : min(max(lo, 0) / T, qt);
      }
      if (lane == 0) first_tab[n] = first;
    }
    __syncthreads();
    first_tile = first_tab;
  }

  // the copy / MMA warps hand registers to the softmax warps (whole groups of four warps switch together)
  if (warp < 4) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::kRegsIO));
  if (warp == 0) {
    // ---------------------------------------------------------------- TMA producer
    // K (with Q at an item's first tile) and V are two independent sequences over the same stream: whichever has a
    // free slot is fetched next, so the K tiles run as far ahead as their ring allows.
    if (lane == 0) {
      Cursor ck, cv;
      ck.init(sched, first_tile);
      cv.init(sched, first_tile);
      bool q_done = false;  // Q of ck's item has been requested
      long long t_idle = clock64();
      while (ck.valid || cv.valid) {
        bool progress = false;
        if (ck.valid) {
          const int b = ck.bh / p.H, h = ck.bh % p.H;
          const int qb = ck.ord % C::kQ;
          if (ck.j == ck.j0 && !q_done && mbar_try_wait(&q_empty[qb], ((ck.ord / C::kQ) & 1) ^ 1u)) {
            mbar_expect_tx(&q_full[qb], kTB);
            load_rows<DHP>(q_s + qb * kTB, &tm_q, &q_full[qb], ck.qt * T, h, b);
            q_done = true;
            progress = true;
          }
          const int st = ck.g % C::kK;
          if ((ck.j > ck.j0 || q_done) && mbar_try_wait(&k_empty[st], ((ck.g / C::kK) & 1) ^ 1u)) {
            mbar_expect_tx(&k_full[st], kTB);
            load_rows<DHP>(k_s + st * kTB, &tm_k, &k_full[st], ck.j * T, h, b);
            ck.advance(sched);
            q_done = false;
            progress = true;
          }
        }
        if (cv.valid) {
          const int st = cv.g % C::kV;
          if (mbar_try_wait(&v_empty[st], ((cv.g / C::kV) & 1) ^ 1u)) {
            mbar_expect_tx(&v_full[st], kTB);
            load_rows<DHP>(v_s + st * kTB, &tm_v, &v_full[st], cv.j * T, cv.bh % p.H, cv.bh / p.H);
            cv.advance(sched);
            progress = true;
          }
        }
        if (progress) {
          t_idle = clock64();
        } else {
          if (*abort_flag) break;
          if (clock64() - t_idle > kWaitLimitCycles) {
            *abort_flag = 1;
            record_fault(p.fault, 0x1101u);
            break;
          }
        }
      }
    }
  } else if (warp == 1) {
    // ---------------------------------------------------------------- MMA issuer, scores: S = Q K^T
    // every lane walks the stream and waits (addresses and descriptors stay warp-uniform); an elected lane issues
    constexpr uint32_t idesc_s = idesc_bf16_f32(T, T, false, false);
    Cursor a;
    a.init(sched, first_tile);
    bool ok = true;
    while (a.valid && ok) {
      const int st = a.g % C::kK;
      const int qb = a.ord % C::kQ;
      const int sb = a.g % kSBufs;
      bool w = true;
      if (a.j == a.j0) w = mbar_wait(&q_full[qb], (a.ord / C::kQ) & 1, ctx, 0x1201u);
      if (w) w = mbar_wait(&k_full[st], (a.g / C::kK) & 1, ctx, 0x1202u);
      if (w) w = mbar_wait(&s_free[sb], ((a.g / kSBufs) & 1) ^ 1u, ctx, 0x1203u);  // tile g - 2 has been read out
      ok = __all_sync(0xffffffffu, w);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t qa = smem_u32(q_s + qb * kTB), ka = smem_u32(k_s + st * kTB);
      const uint32_t dst = tmem + sb * T;
#pragma unroll
      for (int k16 = 0; k16 < DHP / 16; ++k16)
        mma_bf16_ss_elect(dst, desc_kmajor(qa, k16), desc_kmajor(ka, k16), idesc_s, k16 > 0);
      mma_commit_elect(&s_full[sb]);
      mma_commit_elect(&k_empty[st]);
      if (a.j == a.qt) mma_commit_elect(&q_empty[qb]);
      a.advance(sched);
    }
  } else if (warp == 2) {
    // ---------------------------------------------------------------- MMA issuer, output: O_x += P[:, c] V[c, :]
    constexpr uint32_t idesc_o = idesc_bf16_f32(T, DHP, false, true);
    constexpr int kPerBlock = T / 16 / C::kNC;  // K steps of a column block
    Cursor b;
    b.init(sched, first_tile);
    bool ok = true;
    while (b.valid && ok) {
      const int st = b.g % C::kV;
      const bool first = b.j - b.j0 < C::kG;  // the group's first tile of the item: fresh accumulators ...
      bool w = mbar_wait(p_ready, b.g & 1, ctx, 0x1204u) &&
               mbar_wait(&v_full[st], (b.g / C::kV) & 1, ctx, 0x1205u);
      if (w && first) w = mbar_wait(o_free, (b.ord & 1) ^ 1u, ctx, 0x1206u);  // ... once the previous item has been read out
      ok = __all_sync(0xffffffffu, w);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t pa = smem_u32(p_s), va = smem_u32(v_s + st * kTB);
#pragma unroll
      for (int part = 0; part < kParts; ++part)
#pragma unroll
        for (int k16 = 0; k16 < T / 16; ++k16)
          mma_bf16_ss_elect(tmem + kColO + ((b.g % C::kG) * C::kNC + k16 / kPerBlock) * DHP,
                            desc_kmajor(pa + part * kPBytes, k16), desc_rows_as_k(va, k16), idesc_o,
                            (part > 0 || k16 % kPerBlock > 0 || !first) ? 1u : 0u);
      mma_commit_elect(&o_full[b.g % C::kG]);
      mma_commit_elect(&v_empty[st]);
      b.advance(sched);
    }
  } else if (warp >= 4) {
    // ---------------------------------------------------------------- softmax warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::kRegsSoftmax));
    constexpr int kCW = C::kCW, kWords = kCW / 32;
    const int quarter = warp & 3;                  // tensor-memory lane quarter this warp may read
    const int grp = (warp - 4) / C::kGroupWarps;   // this group handles the stream's tiles with g % kG == grp
    const int cb = ((warp - 4) >> 2) % C::kNC;     // its column block
    const int row = quarter * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(quarter * 32) << 16;
    const uint32_t t_o = tmem + lane_base + kColO;
    const uint32_t t_own = t_o + (grp * C::kNC + cb) * DHP;
    const float f_eval = p.dr.train ? 1.f : p.dr.eval_scale;  // evaluation: P * (1 - p), applied to the final rows
    const uint32_t thr_hi = p.dr.thr16 << 16;
    const float sc = p.scale_log2;
    const int ntri = p.nq * (p.nq + 1) / 2;
    // float32 probabilities are kept at most 1 (the reference exponent is exceeded by less than 2^8, see below), so that a
    // sum with V overflows no earlier than one of the exact probabilities would
    constexpr float kShift = -8.f;

    Cursor c;
    c.init(sched, first_tile);
    bool ok = true;
    // reference (score units) and sum of 2^((s - m_ref) sc + shift) of this group's tiles of the item, this column block; its
    // true row maximum
    float m_ref = -INFINITY, l = 0.f, m_true = -INFINITY;

    while (c.valid && ok) {
      const int q_row = c.qt * T + row;
      const bool last = c.j == c.qt;
      const bool mine = c.g % C::kG == grp;
      if (!mine && !last) {
        c.advance(sched);
        continue;
      }
      const int first_key = p.kstart != nullptr && q_row < p.S
                                ? __ldg(p.kstart + static_cast<int64_t>(c.bh / p.H) * p.S + q_row) : 0;
      if (mine) {
        const int sb = c.g % kSBufs;
        const bool fresh = c.j - c.j0 < C::kG;
        // what does not wait for the scores: the keep flags of this thread's columns
        uint32_t keepw[kWords];
#pragma unroll
        for (int w = 0; w < kWords; ++w)
          if (MODE == 1)
            keepw[w] = keep_word(rk_s, (static_cast<uint64_t>(c.bh) * p.S + q_row) * p.S + static_cast<uint64_t>(c.j * T + cb * kCW + 32 * w),
                                 p.dr.stream_id, thr_hi);
        if (MODE == 2) {
          const uint2 kb = __ldg(reinterpret_cast<const uint2*>(p.keep_bits) +
                                 ((static_cast<int64_t>(c.bh) * ntri + c.qt * (c.qt + 1) / 2 + c.j) * T + row) * 2 + cb);
          keepw[0] = kb.x;
          keepw[1] = kb.y;
        }
        ok = mbar_wait(&s_full[sb], (c.g / kSBufs) & 1, ctx, 0x1303u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after_sync();
        // The scores are read twice, 32 columns at a time, for the maximum and for the exponentials: 64 live scores a thread
        // do not fit the 104 registers of four warps a scheduler.
        const uint32_t t_s = tmem + lane_base + sb * T + cb * kCW;
        const bool edge = last || p.kstart != nullptr;
        auto load_scores = [&](int w, float (&s)[32]) {
          tmem_ld_32x32f(t_s + 32 * w, s);
          tmem_ld_wait();
          if (edge) {  // keys after the row (diagonal tile) and before its document
            const int k0 = c.j * T + cb * kCW + 32 * w;  // first key of the word
            const uint32_t valid = range_bits(first_key - k0, q_row - k0);
            if (__any_sync(0xffffffffu, valid != 0xffffffffu)) {
#pragma unroll
              for (int i = 0; i < 32; ++i)
                if (((valid >> i) & 1u) == 0u) s[i] = -INFINITY;
            }
          }
        };
        float mp[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};  // four independent chains of three-input maxima
#pragma unroll
        for (int w = 0; w < kWords; ++w) {
          float s[32];
          load_scores(w, s);
#pragma unroll
          for (int i = 0; i < 32; i += 8)
#pragma unroll
            for (int k = 0; k < 4; ++k) mp[k] = max3(mp[k], s[i + 2 * k], s[i + 2 * k + 1]);
        }
        const float mloc = fmaxf(fmaxf(mp[0], mp[1]), fmaxf(mp[2], mp[3]));
        // The reference only moves when the row maximum outgrows it by more than 2^8: probabilities then stay below 256
        // times the shift (same relative precision in any scale) and the accumulator in tensor memory is rescaled rarely.
        // Any reference gives the same quotient sum(P V) / sum(P).
        bool grow = false;
        if (fresh) {
          m_ref = mloc;
          m_true = mloc;
          l = 0.f;
        } else {
          grow = (mloc - m_ref) * sc > 8.f;  // (both -inf: not a number, no growth)
          m_true = fmaxf(m_true, mloc);
        }
        // The P buffer is free once the output MMAs of tile g - 1 are done. (A wait can only tell a phase from the one before
        // it: the group waits for every tile of its own, and where there are two groups for every tile of the other.)
        ok = mbar_wait(&o_full[grp], ((c.g / C::kG) & 1) ^ 1u, ctx, 0x1302u);
        if (C::kG > 1 && ok && c.g > 0)
          ok = mbar_wait(&o_full[(c.g - 1) % C::kG], ((c.g - 1) / C::kG) & 1, ctx, 0x1302u);
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        if (__any_sync(0xffffffffu, grow)) {  // rare: bring the accumulated rows to the new reference
          tc_fence_after_sync();
          const float alpha = grow ? ex2_approx((m_ref - mloc) * sc) : 1.f;
          if (grow) {
            m_ref = mloc;
            l *= alpha;
          }
#pragma unroll
          for (int x = 0; x < DHP; x += 32) {
            uint32_t t[32];
            tmem_ld_32x32(t_own + x, t);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 32; ++i) t[i] = __float_as_uint(__uint_as_float(t[i]) * alpha);
            tmem_st_32x32(t_own + x, t);
          }
          tmem_st_wait();
        }
        // (a row that has met no key of its own yet carries m_ref = -inf; its scores are all -inf too and must give 0)
        const float ref = m_ref == -INFINITY ? 0.f : m_ref;
        const uint64_t sc2 = pack2(sc, sc), sh2 = pack2(kShift, kShift);
        const uint64_t nm2 = pack2(-ref, -ref);
        uint64_t rp[2] = {0ull, 0ull};  // two packed running sums (four chains)
#pragma unroll
        for (int w = 0; w < kWords; ++w) {
          float s[32];
          load_scores(w, s);
          if (w == kWords - 1) {  // the scores are in registers: the buffer may take tile g + 2
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(&s_free[sb]);
          }
#pragma unroll
          for (int i8 = 0; i8 < 32; i8 += 8) {
#pragma unroll
            for (int i = i8; i < i8 + 8; i += 2) {  // exp2(-inf) = 0 takes care of the masked columns
              const uint64_t x = pack2(s[i], s[i + 1]);
              float a, b;
              unpack2(fma2(add2(x, nm2), sc2, sh2), a, b);
              a = ex2_approx(a);
              b = ex2_approx(b);
              rp[(i >> 1) & 1] = add2(rp[(i >> 1) & 1], pack2(a, b));
              s[i] = a;
              s[i + 1] = b;
            }
            uint32_t pw[kParts][4];
            split8<kParts>(s + i8, pw);
            if (MODE != 0) {
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                const uint32_t m = pair_mask(keepw[w], (i8 >> 1) + i);
#pragma unroll
                for (int part = 0; part < kParts; ++part) pw[part][i] &= m;
              }
            }
            store8<kParts>(p_s, row, (cb * kCW + 32 * w + i8) >> 3, pw);
          }
        }
        {
          float a, b;
          unpack2(add2(rp[0], rp[1]), a, b);
          l += a + b;
        }
        {  // this warp's share of the V tile: elements that are not finite must not meet masked probabilities
          const int st = c.g % C::kV;
          ok = mbar_wait(&v_full[st], (c.g / C::kV) & 1, ctx, 0x1307u);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          uint8_t* vt = v_s + st * kTB + (warp - 4) % C::kGroupWarps * (kTB / C::kGroupWarps) + lane * 16;
          bool bad = false;
#pragma unroll
          for (int x = 0; x < kTB / C::kGroupWarps; x += 512) bad = zero_nonfinite(vt + x) || bad;
          if (bad) bad_v[c.ord & 1] = c.ord + 1;
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(p_ready);
      }
      if (last) {  // the item ends with this tile: its group merges the states of all and writes the rows
        ok = mbar_wait(o_free, (c.ord & 1) ^ 1u, ctx, 0x1306u);  // the previous item's states have been read
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        float* own = stats + (grp * C::kNC + cb) * 3 * T + row;
        own[0] = m_ref;
        own[T] = l;
        own[2 * T] = m_true;
        m_ref = m_true = -INFINITY;
        l = 0.f;
        __syncwarp();
        if (lane == 0) mbar_arrive(stats_full);
      }
      if (last && mine) {
        ok = mbar_wait(stats_full, c.ord & 1, ctx, 0x1304u) &&
             mbar_wait(&o_full[grp], (c.g / C::kG) & 1, ctx, 0x1305u);  // (of the last tile, and so of all before it)
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) break;
        tc_fence_after_sync();
        const bool odd = __any_sync(0xffffffffu, bad_v[c.ord & 1] == c.ord + 1);  // (read before o_free lets the slot go)
        const bool single = c.j == c.j0;  // the other group had no tile of this item: its accumulators hold anything
        float mx = -INFINITY, mt = -INFINITY, f[C::kAcc], lsum = 0.f;
#pragma unroll
        for (int x = 0; x < C::kAcc; ++x) {
          f[x] = stats[(x * 3 + 0) * T + row];
          mx = fmaxf(mx, f[x]);
          mt = fmaxf(mt, stats[(x * 3 + 2) * T + row]);
        }
#pragma unroll
        for (int x = 0; x < C::kAcc; ++x) {  // (a block that met no key of this row: -inf - -inf is not a number)
          f[x] = f[x] == -INFINITY ? 0.f : ex2_approx((f[x] - mx) * sc);
          lsum = fmaf(stats[(x * 3 + 1) * T + row], f[x], lsum);
        }
        const bool none = first_key > q_row;  // the row attends nothing: zero output, neutral statistics
        const float inv = none ? 0.f : f_eval / lsum;
        constexpr int kOut = DHP / C::kNC;  // columns of the rows that this warp writes
        __nv_bfloat16* dst = views.o.row(c.bh / p.H, c.bh % p.H, q_row);
#pragma unroll
        for (int x0 = 0; x0 < kOut; x0 += 16) {
          const int col = cb * kOut + x0;
          float o[16];
#pragma unroll
          for (int i = 0; i < 16; ++i) o[i] = 0.f;
#pragma unroll
          for (int x = 0; x < C::kAcc; ++x) {
            if (single && x / C::kNC != grp) continue;
            uint32_t t[16];
            tmem_ld_32x16(t_o + x * DHP + col, t);
            tmem_ld_wait();
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] = fmaf(__uint_as_float(t[i]), f[x], o[i]);
          }
          if (x0 + 16 == kOut) {
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(o_free);  // the next item may overwrite the accumulators
          }
          if (odd) {
            float t[16];
#pragma unroll
            for (int i = 0; i < 16; ++i) t[i] = 0.f;
            add_nonfinite_v(t, views.q, views.k, views.v, p, rk_s, MODE, c.bh, q_row, first_key, q_row < p.S && !none, col, mt);
#pragma unroll
            for (int i = 0; i < 16; ++i) o[i] += t[i];
          }
          if (q_row < p.S) {
#pragma unroll
            for (int c8 = 0; c8 < 2; ++c8) {
              float t[8];
#pragma unroll
              for (int i = 0; i < 8; ++i) t[i] = none ? 0.f : o[c8 * 8 + i] * inv;
              if (col + c8 * 8 < p.D) Elem<__nv_bfloat16>::store_vec(dst + col + c8 * 8, t);
            }
          }
        }
        if (cb == 0 && q_row < p.S) {
          const int64_t ri = static_cast<int64_t>(c.bh) * p.S + q_row;
          row_max[ri] = none ? 0.f : mt * p.scale;  // acts0: row maximum of the scaled scores
          // acts1: sum of exp(score - maximum); every score -inf: no reference to move from
          row_sum[ri] = none ? 1.f : (mx == -INFINITY ? lsum : lsum * ex2_approx((mx - mt) * sc - kShift));
        }
      }
      c.advance(sched);
    }
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

// Keep flags of the attention-probability dropout for one call, computed once and shared by the forward and the
// backward kernel: word c of the uint4 at ((bh * ntri + qt (qt + 1) / 2 + kt) * 128 + row) holds the flags of
// columns 32 c .. 32 c + 31 of row `row` of tile (qt, kt); ntri = nq (nq + 1) / 2. One thread per word.
__global__ void __launch_bounds__(512)
attn_keep_bits_kernel(uint32_t* __restrict__ bits, const AttnDropout dr, int S, int nq) {
  grid_dep_sync();
  __shared__ uint32_t rk_s[20];
  if (threadIdx.x == 0) philox_round_keys(dr.seed, rk_s);
  __syncthreads();
  uint32_t rk[20];  // in registers: the kernel is bound by its integer instructions, keys as plain operands
#pragma unroll
  for (int i = 0; i < 20; ++i) rk[i] = rk_s[i];
  // one block per tile (its position is decoded once), one thread per word: 128 rows x 4 words
  const int ntri = nq * (nq + 1) / 2;
  const int64_t tile = blockIdx.x;  // bh * ntri + tri
  const int64_t bh = tile / ntri;
  const int tri = static_cast<int>(tile % ntri);
  int qt = static_cast<int>((sqrtf(8.f * tri + 1.f) - 1.f) * 0.5f);
  while ((qt + 1) * (qt + 2) / 2 <= tri) ++qt;
  while (qt * (qt + 1) / 2 > tri) --qt;
  const int kt = tri - qt * (qt + 1) / 2;
  const int cc = threadIdx.x & 3, row = threadIdx.x >> 2;
  const uint64_t idx0 = (static_cast<uint64_t>(bh) * S + static_cast<uint64_t>(qt) * T + row) * S +
                        static_cast<uint64_t>(kt) * T + cc * 32;
  // four Philox calls (round keys from the kernel parameters), eight 16-bit lanes each: bit e of a call's byte is set
  // when lane e (low half of word e / 2 for even e, high half for odd e) is >= the threshold
  const uint32_t thr_hi = dr.thr16 << 16;
  uint32_t word = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t w[4];
    philox_rk(rk, (idx0 >> 3) + q, dr.stream_id, w);
    word |= keep_flags8(w, thr_hi) << (8 * q);
  }
  if (const uint32_t shift = static_cast<uint32_t>(idx0) & 7u; shift != 0u) {  // rows that start inside a call
    uint32_t w[4];
    philox_rk(rk, (idx0 >> 3) + 4, dr.stream_id, w);
    word = __funnelshift_r(word, keep_flags8(w, thr_hi), shift);
  }
  bits[tile * 512 + threadIdx.x] = word;
}

template <int DHP>
int launch_fwd(const CUtensorMap& tq, const CUtensorMap& tk, const CUtensorMap& tv, const FwdViews& views, float* row_max,
               float* row_sum, const AttnParams& p, int mode, cudaStream_t st) {
  using C = Cfg<DHP>;
  using Kern = void (*)(const CUtensorMap, const CUtensorMap, const CUtensorMap, const FwdViews, float*, float*,
                        const AttnParams, const Sched);
  static const Kern kerns[3] = {attn_fwd_ws_kernel<DHP, 0>, attn_fwd_ws_kernel<DHP, 1>,
                                attn_fwd_ws_kernel<DHP, 2>};
  const Kern kern = kerns[mode];
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes) != cudaSuccess) {
    (void)cudaGetLastError();
    return PTJ_ERR_LAUNCH;
  }
  Sched s;
  const int grid = make_sched(&s, p);
  launch_k(kern, grid, C::kThreads, C::kSmemBytes, st, tq, tk, tv, views, row_max, row_sum, p, s);
  PTJ_CHECK_LAUNCH();
  return PTJ_OK;
}

}  // namespace

size_t attn_keep_bits_bytes(const ptj_attn_shape& sh) {
  const int64_t nq = ceil_div(sh.seq, T);
  return static_cast<size_t>(sh.batch * sh.heads * (nq * (nq + 1) / 2) * T) * 16;
}

int attn_keep_bits_tc(uint32_t* bits, const ptj_attn_shape& sh, const AttnDropout& dr, cudaStream_t st) {
  const int64_t tiles = static_cast<int64_t>(attn_keep_bits_bytes(sh) / 2048);
  launch_k(attn_keep_bits_kernel, static_cast<unsigned>(tiles), 512, 0, st, bits, dr, static_cast<int>(sh.seq),
           static_cast<int>(ceil_div(sh.seq, T)));
  PTJ_CHECK_LAUNCH();
  return PTJ_OK;
}

int attn_fwd_tc(const void* q, const void* k, const void* v, void* o, float* row_max, float* row_sum,
                const uint32_t* keep_bits, const int32_t* row_kstart, const ptj_attn_shape& sh, const AttnDropout& dr,
                cudaStream_t st) {
  if (attn_bf16_probabilities(sh)) return attn_fwd_tc64(q, k, v, o, row_max, row_sum, keep_bits, row_kstart, sh, dr, st);
  CUtensorMap tq, tk, tv;
  if (!make_map(&tq, q, sh, sh.q_strides) || !make_map(&tk, k, sh, sh.k_strides) || !make_map(&tv, v, sh, sh.v_strides))
    return PTJ_ERR_LAUNCH;
  AttnParams p = make_params(sh, dr);
  if (p.fault == nullptr) return PTJ_ERR_DEVICE;
  p.keep_bits = reinterpret_cast<const uint4*>(keep_bits);
  p.kstart = row_kstart;
  const bool masked = dr.train && dr.thr16 != 0u;
  const int mode = !masked ? 0 : (keep_bits != nullptr ? 2 : 1);
  const FwdViews views{make_view(q, sh.q_strides), make_view(k, sh.k_strides), make_view(v, sh.v_strides),
                       make_view(o, sh.o_strides)};
  if (sh.d_head > 64) return launch_fwd<128>(tq, tk, tv, views, row_max, row_sum, p, mode, st);
  return launch_fwd<64>(tq, tk, tv, views, row_max, row_sum, p, mode, st);
}

}  // namespace ptj
