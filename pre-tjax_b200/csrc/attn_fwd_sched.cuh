// The stream of tiles that a thread block of the tcgen05 attention forward kernels walks.
#pragma once
#include "attn_tc_dev.cuh"

namespace ptj {
namespace attn_tc {

struct Sched {
  int total, rounds, nq, BH;
  uint32_t bh_magic;  // ceil(2^32 / BH): x / BH == umulhi(x, bh_magic) for every x the kernel meets (checked on the host)
};

// Position in the stream of (item, kv tile) pairs of one thread block; every role walks the same stream.
// first_tile (row_kstart): per round of this block, the first KV tile its item needs (keys before the first key of every
// row of the query tile are masked anyway: those tiles are skipped); nullptr = every item starts at tile 0.
constexpr int kMaxRoundsTabled = 32;
struct Cursor {
  int n, ord, qt, bh, j, j0, g;
  bool valid;
  const int* first_tile;
  __device__ __forceinline__ void next_item(const Sched& s) {
    valid = false;
    while (++n < s.rounds) {
      const int pos = (n & 1) ? static_cast<int>(gridDim.x) - 1 - static_cast<int>(blockIdx.x) : static_cast<int>(blockIdx.x);
      const int sp = n * static_cast<int>(gridDim.x) + pos;
      if (sp < s.total) {
        const int t = s.BH == 1 ? sp : static_cast<int>(__umulhi(static_cast<uint32_t>(sp), s.bh_magic));  // sp / BH
        qt = s.nq - 1 - t;
        bh = sp - t * s.BH;
        j0 = first_tile != nullptr ? first_tile[n] : 0;
        j = j0;
        ++ord;
        valid = true;
        return;
      }
    }
  }
  __device__ __forceinline__ void init(const Sched& s, const int* first = nullptr) {
    n = -1; ord = -1; g = 0; qt = 0; bh = 0; j = 0; j0 = 0;
    first_tile = first;
    next_item(s);
  }
  __device__ __forceinline__ void advance(const Sched& s) {
    ++g;
    if (j == qt) next_item(s); else ++j;
  }
};

// Grid (returned) and stream of one block per SM over nq query tiles of BH heads.
inline int make_sched(Sched* s, const AttnParams& p) {
  s->nq = p.nq;
  s->BH = p.BH;
  s->total = p.nq * p.BH;
  const int grid = s->total < kNumSMs ? s->total : kNumSMs;
  s->rounds = (s->total + grid - 1) / grid;
  s->bh_magic = static_cast<uint32_t>(((1ull << 32) + s->BH - 1) / s->BH);
  return grid;
}

}  // namespace attn_tc
}  // namespace ptj
