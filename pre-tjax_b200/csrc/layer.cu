// One transformer layer, forward and backward, as a sequence of this library's own entry points: host code only. A step
// issued from Python pays some 12 us per kernel for tensors, views and argument conversion; from here a launch costs 2 to 3,
// which is what small models and short rows are bound by. The sequence is the one the kernels were written for: QKV in one
// product, bias / GELU / dropout / residual in product epilogues, pairs of weight gradients in one launch, dropout of a
// residual branch's gradient and its column sums in the LayerNorm backward (model_triton.py:2343-2410, 2545-2581).
#include <math.h>

#include "attn_common.cuh"

using namespace ptj;

namespace {

// what the steps of one layer share
struct Layer {
  const ptj_layer_shape& d;
  int64_t T, D, F;
  int dtype;
  cudaStream_t st;
  float* ws;
  size_t ws_n;
  explicit Layer(const ptj_layer_shape& s, void* workspace, size_t bytes, void* stream)
      : d(s), T(s.batch * s.seq), D(s.dim), F(s.ffn), dtype(s.dtype), st(static_cast<cudaStream_t>(stream)),
        ws(static_cast<float*>(workspace)), ws_n(bytes / 4) {}

  ptj_attn_shape attn_shape() const {  // columns of the projection: (head, q/k/v, d_head)
    const int64_t dh = D / d.heads, S = d.seq;
    ptj_attn_shape a{};
    a.batch = d.batch; a.heads = d.heads; a.seq = S; a.d_head = dh;
    const int64_t qkv[3] = {S * 3 * D, 3 * dh, 3 * D}, o[3] = {S * D, dh, D};
    for (int i = 0; i < 3; ++i) {
      a.q_strides[i] = a.k_strides[i] = a.v_strides[i] = qkv[i];
      a.o_strides[i] = o[i];
    }
    return a;
  }

  // C[T, N] = A[T, K] op(W): W stored [N, K] (forward) or [K, N] (input gradient)
  int product(const void* a, const void* w, void* c, int64_t N, int64_t K, bool w_kmajor, int epilogue = PTJ_EPI_NONE,
              const float* bias = nullptr, const void* aux = nullptr, void* aux_out = nullptr,
              const ptj_dropout_args* drop = nullptr, int split = 1) const {
    return ptj_gemm(a, w, c, bias, aux, aux_out, T, N, K, K, w_kmajor ? K : N, N, 1, w_kmajor, dtype, dtype, epilogue, drop,
                    split, ws, ws_n, st);
  }
  bool tail(int64_t N, int64_t K) const { return dtype == PTJ_BF16 && ptj_gemm_tail_split_floats(T, N, K) > 0; }
  int dgrad(const void* dy, const void* w, void* dx, int64_t N, int64_t K) const {
    return product(dy, w, dx, N, K, false, PTJ_EPI_NONE, nullptr, nullptr, nullptr, nullptr, tail(N, K) ? PTJ_SPLIT_TAIL : 1);
  }

  // K parts of a weight gradient: rounds of the 74 thread-block pairs, each 1 / S long, plus a charge per part for its
  // float32 partial output (fitted to a sweep over the GPT-2 small shapes at K = 8192: 1.7 us per part of a 9.4 MB output
  // against 55 us for a full-K tile). unsplit_free: a single part writes no partial output.
  int split_for(int64_t tiles, double out_mb, bool unsplit_free) const {
    const int64_t most = T / 64 / 4 > 1 ? T / 64 / 4 : 1;
    int best = 1;
    double best_cost = INFINITY;
    for (int s = 1; s <= 8 && s <= most; ++s) {
      const double charge = unsplit_free && s == 1 ? 0.0 : 0.0032 * out_mb * (8192.0 / static_cast<double>(T)) * s;
      const double cost = static_cast<double>((tiles * s + 73) / 74) / s + charge;
      if (cost < best_cost - 1e-9) {
        best = s;
        best_cost = cost;
      }
    }
    return best;
  }
  static int64_t tiles(int64_t M, int64_t N) { return ceil_div(M, 256) * ceil_div(N, 256); }
  int wgrad_parts(int64_t M, int64_t N) const {
    return dtype == PTJ_BF16 ? split_for(tiles(M, N), static_cast<double>(M * N) * 4e-6, false) : 1;
  }
  int pair_parts(int64_t M0, int64_t N0, int64_t M1, int64_t N1) const {
    const int64_t a = M0 * N0, b = M1 * N1;
    return split_for(tiles(M0, N0) + tiles(M1, N1), static_cast<double>(a > b ? a : b) * 4e-6, true);
  }
  // out[M, N] = dy[T, M]^T x[T, N]; the parts' sums go to the workspace (one part where it does not hold them)
  int wgrad(const void* dy, const void* x, float* out, int64_t M, int64_t N) const {
    const int parts = wgrad_parts(M, N);
    return ptj_gemm(dy, x, out, nullptr, nullptr, nullptr, M, N, T, M, N, N, 0, 0, dtype, PTJ_F32, PTJ_EPI_NONE, nullptr,
                    static_cast<size_t>(parts) * M * N <= ws_n ? parts : 1, ws, ws_n, st);
  }
  int wgrad2(const void* dy0, const void* x0, float* out0, int64_t M0, int64_t N0, const void* dy1, const void* x1, float* out1,
             int64_t M1, int64_t N1) const {
    if (dtype == PTJ_BF16) {
      int s = pair_parts(M0, N0, M1, N1);
      const size_t off = (static_cast<size_t>(s) * M0 * N0 + 3) & ~static_cast<size_t>(3);
      if (off + static_cast<size_t>(s) * M1 * N1 > ws_n) s = 1;
      const size_t n0 = s > 1 ? static_cast<size_t>(s) * M0 * N0 : 0, n1 = s > 1 ? static_cast<size_t>(s) * M1 * N1 : 0;
      const ptj_gemm_problem p0{dy0, x0, out0, M0, N0, M0, N0, N0, PTJ_F32, PTJ_EPI_NONE, s, n0 ? ws : nullptr, n0};
      const ptj_gemm_problem p1{dy1, x1, out1, M1, N1, M1, N1, N1, PTJ_F32, PTJ_EPI_NONE, s, n1 ? ws + off : nullptr, n1};
      const int rc = ptj_gemm_grouped2(&p0, &p1, T, 0, 0, st);
      if (rc != PTJ_ERR_UNSUPPORTED) return rc;
    }
    const int rc = wgrad(dy0, x0, out0, M0, N0);
    return rc != PTJ_OK ? rc : wgrad(dy1, x1, out1, M1, N1);
  }

  // the LayerNorm backward also writes dropout(dx) for the branch that takes dx next, and that tensor's column sums
  int norm_bwd(const void* dy, const void* x, const float* gamma, const void* dx_add, void* dx, void* dropped, float* dropped_sums,
               float* dgamma, float* dbeta, uint64_t seed) const {
    const size_t n = ptj_layernorm_bwd_scratch_floats(T, D);
    if (n > ws_n) return PTJ_ERR_WORKSPACE;
    if (dropped == nullptr) return ptj_layernorm_bwd(dy, x, gamma, dx_add, dx, dgamma, dbeta, ws, n, T, D, dtype, st);
    return ptj_layernorm_bwd_dropout(dy, x, gamma, dx_add, dx, dropped, dropped_sums, dgamma, dbeta, ws, n, T, D, d.p, d.train, seed,
                                     0, dtype, st);
  }
  int sums(const void* x, float* out, int64_t cols) const {
    const size_t n = ptj_colsum_scratch_floats(T, cols);
    return n > ws_n ? PTJ_ERR_WORKSPACE : ptj_colsum(x, out, ws, n, T, cols, cols, dtype, st);
  }
};

bool shape_ok(const ptj_layer_shape* s) {
  return s != nullptr && s->batch >= 1 && s->seq >= 1 && s->dim >= 1 && s->heads >= 1 && s->ffn >= 1 && s->dim % s->heads == 0 &&
         (s->dtype == PTJ_F32 || s->dtype == PTJ_BF16);
}

#define PTJ_TRY(call)               \
  do {                              \
    const int rc_ = (call);         \
    if (rc_ != PTJ_OK) return rc_;  \
  } while (0)

}  // namespace

extern "C" size_t ptj_layer_workspace_bytes(const ptj_layer_shape* s, int backward, int products) {
  if (!shape_ok(s)) return 0;
  const Layer l(*s, nullptr, 0, nullptr);
  const int64_t T = l.T, D = l.D, F = l.F;
  size_t most = 4;
  auto need = [&](size_t floats) { most = floats > most ? floats : most; };
  if (backward) {
    need(ptj_layernorm_bwd_scratch_floats(T, D));
    need(ptj_colsum_scratch_floats(T, F));
    const ptj_attn_shape a = l.attn_shape();
    // (shapes with float32 probabilities run without it, on the general kernels)
    if (products || attn_bf16_probabilities(a)) need((ptj_attn_bwd_workspace_bytes(&a, s->dtype) + 3) / 4);
  }
  if (!products) return most * sizeof(float);
  if (s->dtype == PTJ_F32) {
    const int64_t n[4] = {3 * D, D, F, D}, k[4] = {D, D, D, F};
    for (int i = 0; i < 4; ++i) {
      need(ptj_gemm_f32_workspace_floats(T, n[i], k[i], 1, 1));
      if (!backward) continue;
      need(ptj_gemm_f32_workspace_floats(T, k[i], n[i], 1, 0));
      need(ptj_gemm_f32_workspace_floats(n[i], k[i], T, 0, 0));
    }
  } else {
    need(ptj_gemm_tail_split_floats(T, D, F));
    if (backward) {
      need(ptj_gemm_tail_split_floats(T, D, 3 * D));
      need(ptj_gemm_tail_split_floats(T, D, D));
      need(static_cast<size_t>(l.pair_parts(D, F, F, D)) * 2 * D * F + 4);
      need(static_cast<size_t>(l.pair_parts(3 * D, D, D, D)) * 4 * D * D + 4);
      need(static_cast<size_t>(l.wgrad_parts(D, F)) * D * F);
      need(static_cast<size_t>(l.wgrad_parts(F, D)) * D * F);
      need(static_cast<size_t>(l.wgrad_parts(3 * D, D)) * 3 * D * D);
      need(static_cast<size_t>(l.wgrad_parts(D, D)) * D * D);
    }
  }
  return most * sizeof(float);
}

extern "C" size_t ptj_layer_keep_bits_bytes(const ptj_layer_shape* s) {
  if (!shape_ok(s) || !s->train || !(s->p > 0.f)) return 0;
  const ptj_attn_shape a = Layer(*s, nullptr, 0, nullptr).attn_shape();
  return ptj_attn_keep_bits_bytes(&a, s->dtype);
}

extern "C" int ptj_layer_fwd(const ptj_layer_shape* s, const ptj_layer_weights* w, const ptj_layer_acts* a, void* x_out,
                             const int32_t* row_kstart, void* workspace, size_t workspace_bytes, void* stream) {
  if (!shape_ok(s) || w == nullptr || a == nullptr || x_out == nullptr) return PTJ_ERR_BAD_SHAPE;
  const Layer l(*s, workspace, workspace_bytes, stream);
  const int64_t T = l.T, D = l.D, F = l.F;
  const size_t es = s->dtype == PTJ_F32 ? 4 : 2;
  const ptj_attn_shape sh = l.attn_shape();
  const int64_t dh = D / s->heads;
  char* qkv = static_cast<char*>(a->qkv);
  PTJ_TRY(ptj_layernorm_fwd(a->x, w->g1, w->b1, a->ln1, T, D, s->dtype, stream));
  PTJ_TRY(l.product(a->ln1, w->w_qkv, a->qkv, 3 * D, D, true));
  if (a->keep_bits != nullptr)  // drawn once, shared by the forward and backward kernels
    PTJ_TRY(ptj_attn_keep_bits(a->keep_bits, &sh, s->p, s->seed_attn, 0, s->dtype, stream));
  PTJ_TRY(ptj_attn_fwd(qkv, qkv + dh * es, qkv + 2 * dh * es, a->attn, a->row_max, a->row_sum, &sh, s->p, s->train, s->seed_attn, 0,
                       a->keep_bits, row_kstart, s->dtype, stream));
  const ptj_dropout_args d1{s->p, s->train, s->seed_res1, 0}, d2{s->p, s->train, s->seed_res2, 0};
  PTJ_TRY(l.product(a->attn, w->w_o, a->x_mid, D, D, true, PTJ_EPI_DROPOUT_RESID, nullptr, a->x, nullptr, &d1));
  PTJ_TRY(ptj_layernorm_fwd(a->x_mid, w->g2, w->b2, a->ln2, T, D, s->dtype, stream));
  PTJ_TRY(l.product(a->ln2, w->w1, a->h_act, F, D, true, PTJ_EPI_GELU, w->b1f, nullptr, a->h_pre));
  return l.product(a->h_act, w->w2, x_out, D, F, true, PTJ_EPI_DROPOUT_RESID, w->b2f, a->x_mid, nullptr, &d2,
                   l.tail(D, F) ? PTJ_SPLIT_TAIL : 1);
}

extern "C" int ptj_layer_bwd_ffn(const ptj_layer_shape* s, const ptj_layer_weights* w, const ptj_layer_acts* a,
                                 const ptj_layer_grads* g, const void* dx, const void* dy, void* dh_pre, void* d_ln, void* dx_out,
                                 void* dy_out, void* workspace, size_t workspace_bytes, void* stream) {
  if (!shape_ok(s) || w == nullptr || a == nullptr || g == nullptr) return PTJ_ERR_BAD_SHAPE;
  const Layer l(*s, workspace, workspace_bytes, stream);
  const int64_t D = l.D, F = l.F;
  // x_out = x_mid + dropout(W2 gelu(W1 ln2(x_mid) + b1f) + b2f)
  PTJ_TRY(l.product(dy, w->w2, dh_pre, F, D, false, PTJ_EPI_GELU_BWD, nullptr, a->h_pre));
  PTJ_TRY(l.sums(dh_pre, g->b1f, F));
  PTJ_TRY(l.wgrad2(dy, a->h_act, g->w2, D, F, dh_pre, a->ln2, g->w1, F, D));
  PTJ_TRY(l.dgrad(dh_pre, w->w1, d_ln, D, F));
  return l.norm_bwd(d_ln, a->x_mid, w->g2, dx, dx_out, dy_out, nullptr, g->g2, g->b2, s->seed_res1);
}

extern "C" int ptj_layer_bwd_attn(const ptj_layer_shape* s, const ptj_layer_weights* w, const ptj_layer_acts* a,
                                  const ptj_layer_grads* g, const void* dx, const void* dy, void* d_attn, void* dqkv, void* d_ln,
                                  void* dx_out, void* dy_out, float* dy_sums, uint64_t seed_below, const int32_t* row_kstart,
                                  void* workspace, size_t workspace_bytes, void* stream) {
  if (!shape_ok(s) || w == nullptr || a == nullptr || g == nullptr) return PTJ_ERR_BAD_SHAPE;
  const Layer l(*s, workspace, workspace_bytes, stream);
  const int64_t D = l.D;
  const size_t es = s->dtype == PTJ_F32 ? 4 : 2;
  const ptj_attn_shape sh = l.attn_shape();
  const int64_t dh = D / s->heads;
  char *q = static_cast<char*>(a->qkv), *dq = static_cast<char*>(dqkv);
  // x_mid = x + dropout(attn(ln1(x)) W_o^T)
  PTJ_TRY(l.dgrad(dy, w->w_o, d_attn, D, D));
  PTJ_TRY(ptj_attn_bwd(d_attn, q, q + dh * es, q + 2 * dh * es, a->attn, a->row_max, a->row_sum, dq, dq + dh * es, dq + 2 * dh * es,
                       &sh, &sh, s->p, s->train, s->seed_attn, 0, a->keep_bits, row_kstart, workspace, workspace_bytes, s->dtype,
                       stream));
  PTJ_TRY(l.wgrad2(dqkv, a->ln1, g->w_qkv, 3 * D, D, dy, a->attn, g->w_o, D, D));
  PTJ_TRY(l.dgrad(dqkv, w->w_qkv, d_ln, D, 3 * D));
  return l.norm_bwd(d_ln, a->x, w->g1, dx, dx_out, dy_out, dy_sums, g->g1, g->b1, seed_below);
}
