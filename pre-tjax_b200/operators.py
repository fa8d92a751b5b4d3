"""Drop-in operator surface: the launcher functions of the reference's Triton path, backed by the sm_100a library.

Names, argument order and return structure follow pre-tjax's ``model_triton.py`` / ``loss_and_optimizer_triton.py``
(cited per function). Tensors are CUDA tensors, float32 or bfloat16; results are fresh tensors, inputs are never
modified. Unlike the reference, no output needs zero-initialisation and nothing uses atomics.

The dropout rate is a module constant, as in the reference (model_torch_func.py:2, model_triton.py:21):
set ``operators.DROPOUT_RATE`` before calling.
"""
from __future__ import annotations

import ctypes
import math
import weakref

import torch

from . import _lib
from ._lib import AttnShape, DropoutArgs, PTJ_BF16, PTJ_F32

DROPOUT_RATE = 0.1
# When set to a list, every tensor-core GEMM appends (start event, stop event, 2*M*N*K, (M, N, K, a_kmajor, b_kmajor),
# algorithmic bytes) to it: lets a benchmark attribute device time, FLOPs and bytes to the GEMM kernel without a profiler.
GEMM_PROFILE = None


# ---- plumbing -------------------------------------------------------------------------------------------------------
_DTYPE_CODES = {torch.float32: PTJ_F32, torch.bfloat16: PTJ_BF16}


def _dt(t: torch.Tensor) -> int:
    code = _DTYPE_CODES.get(t.dtype)
    if code is None:
        raise TypeError(f"unsupported dtype {t.dtype}: the kernels take float32 or bfloat16")
    return code


def _cuda(t: torch.Tensor, name: str = "tensor") -> torch.Tensor:
    if not t.is_cuda:
        raise RuntimeError(f"{name} must live on a CUDA device: there is no CPU implementation")
    return t if t.is_contiguous() else t.contiguous()


def _f32(t: torch.Tensor) -> torch.Tensor:
    t = _cuda(t)
    return t if t.dtype == torch.float32 else t.float()


def _stream() -> int:
    """Handle of the current device's current stream, without building a Stream object (1.3 us of each launch)."""
    return torch._C._cuda_getCurrentRawStream(torch._C._cuda_getDevice())


def _ptr(t) -> int:
    return 0 if t is None else t.data_ptr()


SEED_IS_POINTER = 1 << 63


class SeedRef(int):
    """A seed argument that is the address of a device word (bit 63 set), not a seed value."""


def seed_at(words: torch.Tensor, index: int = 0) -> SeedRef:
    """A seed argument that makes the kernels read the seed from element `index` of a CUDA int64 tensor when they run
    (PTJ_SEED_AT of the C header): lets a recorded step (CUDA graph) be replayed with fresh dropout masks. The tensor
    must stay alive, and hold its final value, whenever a kernel that was given the reference runs."""
    assert words.is_cuda and words.dtype == torch.int64 and 0 <= index < words.numel()
    return SeedRef((words.data_ptr() + 8 * index) | SEED_IS_POINTER)


def _seed(p_gen_aux) -> int:
    """Immediate seeds are 63-bit values: bit 63 marks a device-resident seed (seed_at) and is cleared otherwise."""
    if p_gen_aux is None:
        return 0
    if isinstance(p_gen_aux, SeedRef):
        return int(p_gen_aux)
    return int(p_gen_aux) & (SEED_IS_POINTER - 1)


# ---- LayerNorm ------------------------------------------------------------------------------------------------------
def t_layernorm_fwd_t(layer_params, x: torch.Tensor) -> torch.Tensor:
    """gamma * (x - mean) / unbiased_std + beta over the last dim (model_triton.py:1625-1637)."""
    x = _cuda(x, "x")
    gamma, beta = _f32(layer_params[0]), _f32(layer_params[1])
    y = torch.empty_like(x)
    dim = x.shape[-1]
    rows = x.numel() // dim if dim else 0
    _lib.check(_lib.lib().ptj_layernorm_fwd(_ptr(x), _ptr(gamma), _ptr(beta), _ptr(y), rows, dim, _dt(x), _stream()),
               "ptj_layernorm_fwd")
    return y


def layernorm_bwd(dloss_dx, layer_params, x, want_dx=True, want_dp=True, dx_add=None, dgamma_out=None,
                  dbeta_out=None, dropped=None, dropped_colsum_out=None):
    """Fused LayerNorm backward: (dx or None, dgamma or None, dbeta or None); dx_add is added onto dx.
    dgamma_out / dbeta_out: optional float32 destinations (e.g. views of a flat gradient buffer).
    dropped = (train, seed, p[, stream_id]): additionally return, as a fourth value, dropout(dx) for that mask site
    (what t_dropout of dx would give), written by the same kernel; dropped_colsum_out (float32[dim], needs want_dp)
    receives that tensor's column sums, the bias gradient of the linear layer feeding the dropped branch."""
    x = _cuda(x, "x")
    dy = _cuda(dloss_dx, "dloss_dx")
    if dy.dtype != x.dtype:
        dy = dy.to(x.dtype)
    gamma = _f32(layer_params[0])
    dim = x.shape[-1]
    rows = x.numel() // dim
    dx = torch.empty_like(x) if want_dx else None
    dg = db = scratch = None
    n_scratch = 0
    if want_dp:
        dg = dgamma_out if dgamma_out is not None else x.new_empty(dim, dtype=torch.float32)
        db = dbeta_out if dbeta_out is not None else x.new_empty(dim, dtype=torch.float32)
        n_scratch = _lib.lib().ptj_layernorm_bwd_scratch_floats(rows, dim)
        scratch = x.new_empty(max(n_scratch, 1), dtype=torch.float32)
    if dx_add is not None:
        dx_add = _cuda(dx_add, "dx_add")
    if dropped is not None:
        train, seed, p = dropped[:3]
        stream_id = dropped[3] if len(dropped) > 3 else 0
        dxd = torch.empty_like(x)
        _lib.check(
            _lib.lib().ptj_layernorm_bwd_dropout(_ptr(dy), _ptr(x), _ptr(gamma), _ptr(dx_add), _ptr(dx), _ptr(dxd),
                                                 _ptr(dropped_colsum_out), _ptr(dg), _ptr(db), _ptr(scratch), n_scratch, rows, dim,
                                                 DROPOUT_RATE if p is None else p, int(bool(train)), _seed(seed),
                                                 stream_id, _dt(x), _stream()), "ptj_layernorm_bwd_dropout")
        return dx, dg, db, dxd
    _lib.check(
        _lib.lib().ptj_layernorm_bwd(_ptr(dy), _ptr(x), _ptr(gamma), _ptr(dx_add), _ptr(dx), _ptr(dg), _ptr(db),
                                     _ptr(scratch), n_scratch, rows, dim, _dt(x), _stream()),
        "ptj_layernorm_bwd")
    return dx, dg, db


def t_layernorm_bkwd2_p_t(dloss_dx, layer_params, x):
    """(dgamma, dbeta) (model_triton.py:1710-1726)."""
    _, dg, db = layernorm_bwd(dloss_dx, layer_params, x, want_dx=False, want_dp=True)
    return dg, db


def t_layernorm_bkwd2_x_t(dloss_dx, layer_params, x):
    """dx (model_triton.py:1853-1867)."""
    dx, _, _ = layernorm_bwd(dloss_dx, layer_params, x, want_dx=True, want_dp=False)
    return dx.reshape(dloss_dx.shape)


# ---- GELU -----------------------------------------------------------------------------------------------------------
def t_gelu_fwd_t(x: torch.Tensor) -> torch.Tensor:
    """tanh-GELU (model_triton.py:254-260)."""
    x = _cuda(x, "x")
    y = torch.empty_like(x)
    _lib.check(_lib.lib().ptj_gelu_fwd(_ptr(x), _ptr(y), x.numel(), _dt(x), _stream()), "ptj_gelu_fwd")
    return y


def t_gelu_bkwd2_t(dloss_dx: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """dloss_dx * gelu'(x) (model_triton.py:296-304)."""
    x = _cuda(x, "x")
    dy = _cuda(dloss_dx, "dloss_dx").to(x.dtype)
    out = torch.empty_like(x)
    _lib.check(_lib.lib().ptj_gelu_bwd(_ptr(dy), _ptr(x), _ptr(out), x.numel(), _dt(x), _stream()), "ptj_gelu_bwd")
    return out


# ---- dropout --------------------------------------------------------------------------------------------------------
def dropout(x, train, seed, stream_id=0, residual=None, p=None):
    x = _cuda(x, "x")
    if residual is not None:
        residual = _cuda(residual, "residual").to(x.dtype)
    y = torch.empty_like(x)
    p = DROPOUT_RATE if p is None else p
    _lib.check(_lib.lib().ptj_dropout(_ptr(x), _ptr(residual), _ptr(y), x.numel(), p, int(bool(train)), _seed(seed),
                                      stream_id, _dt(x), _stream()), "ptj_dropout")
    return y


def t_dropout_fwd_t(x: torch.Tensor, train=True, p_gen_aux=None) -> torch.Tensor:
    """x * mask in training (keep probability 1 - DROPOUT_RATE, no rescale), x * (1 - DROPOUT_RATE) otherwise
    (model_triton.py:1496-1506). The mask is a pure function of (p_gen_aux, element index)."""
    return dropout(x, train, p_gen_aux)


def t_dropout_bkwd2_t(dloss_dx: torch.Tensor, x: torch.Tensor, train=True, p_gen_aux=None) -> torch.Tensor:
    """The same mask applied to the gradient (model_triton.py:1562-1572); x only fixes the shape."""
    return dropout(dloss_dx, train, p_gen_aux)


# ---- log-softmax ------------------------------------------------------------------------------------------------------
def t_log_softmax_fwd_t(x: torch.Tensor) -> torch.Tensor:
    """log-softmax over the last dim, any row length (model_triton.py:62-72)."""
    x = _cuda(x, "x")
    y = torch.empty_like(x)
    cols = x.shape[-1]
    rows = x.numel() // cols
    _lib.check(_lib.lib().ptj_log_softmax_fwd(_ptr(x), _ptr(y), rows, cols, cols, cols, _dt(x), _stream()),
               "ptj_log_softmax_fwd")
    return y


def t_log_softmax_bkwd2_t(dloss_dx: torch.Tensor, x: torch.Tensor) -> torch.Tensor:
    """dloss_dx - softmax(x) * sum(dloss_dx) (model_triton.py:153-164)."""
    x = _cuda(x, "x")
    dy = _cuda(dloss_dx, "dloss_dx").to(x.dtype)
    dx = torch.empty_like(x)
    cols = x.shape[-1]
    rows = x.numel() // cols
    _lib.check(_lib.lib().ptj_log_softmax_bwd(_ptr(dy), _ptr(x), _ptr(dx), rows, cols, cols, _dt(x), _stream()),
               "ptj_log_softmax_bwd")
    return dx.reshape(dloss_dx.shape)


SPLIT_TAIL = -1  # ptj_gemm's split_k value "split the rows of a mostly-empty last round of tiles over K"


# ---- GEMM -----------------------------------------------------------------------------------------------------------
def gemm(a, b, *, a_kmajor=True, b_kmajor=True, M=None, N=None, K=None, lda=None, ldb=None, out=None, out_dtype=None,
         ldc=None, bias=None, epilogue=_lib.EPI_NONE, aux=None, aux_out=None, dropout_args=None, split_k=1,
         workspace=None):
    """C[M,N] = op(A) op(B) through ptj_gemm. a_kmajor: A stored [M,K]; else [K,M]. b_kmajor: B stored [N,K]; else [K,N]."""
    dtype = a.dtype
    if dtype != b.dtype:
        raise TypeError("operands of a GEMM must share a dtype")
    lib = _lib.lib()
    if M is None:
        M, K = (a.shape[0], a.shape[1]) if a_kmajor else (a.shape[1], a.shape[0])
    if N is None:
        N = b.shape[0] if b_kmajor else b.shape[1]
    lda = a.stride(0) if lda is None else lda
    ldb = b.stride(0) if ldb is None else ldb
    if out is None:
        out = a.new_empty((M, N), dtype=out_dtype)
    ldc = out.stride(0) if ldc is None else ldc
    ws_n = 0
    if split_k > 1 or split_k == SPLIT_TAIL:
        if dtype != torch.bfloat16:
            split_k = 1
        else:
            ws_n = split_k * M * N if split_k > 1 else lib.ptj_gemm_tail_split_floats(M, N, K)
            if ws_n == 0:
                split_k = 1  # this shape has no bad last round
            elif workspace is None or workspace.numel() < ws_n:
                workspace = torch.empty(ws_n, device=a.device, dtype=torch.float32)
    if dtype == torch.float32 and out.dtype == torch.float32:
        # bf16 planes of both operands (and K parts): with them the product runs on the tensor cores, at float32 accuracy
        ws_n = lib.ptj_gemm_f32_workspace_floats(M, N, K, int(a_kmajor), int(b_kmajor))
        if ws_n and (workspace is None or workspace.numel() < ws_n):
            try:
                workspace = torch.empty(ws_n, device=a.device, dtype=torch.float32)
            except torch.OutOfMemoryError:  # 6 bytes per operand element: a product that fits without them still runs
                workspace = None
    dargs = None
    if dropout_args is not None:
        p, train, seed, sid = dropout_args
        dargs = ctypes.byref(DropoutArgs(p, int(bool(train)), _seed(seed), sid))
    prof = GEMM_PROFILE if (GEMM_PROFILE is not None and a.dtype == torch.bfloat16) else None
    if prof is not None:
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
    rc = lib.ptj_gemm(a.data_ptr(), b.data_ptr(), out.data_ptr(), None if bias is None else bias.data_ptr(),
                      None if aux is None else aux.data_ptr(), None if aux_out is None else aux_out.data_ptr(), M, N, K,
                      lda, ldb, ldc, a_kmajor, b_kmajor, _dt(a), _dt(out), epilogue, dargs, split_k,
                      None if workspace is None else workspace.data_ptr(),
                      0 if workspace is None else workspace.numel(), _stream())
    if rc != 0:
        _lib.check(rc, "ptj_gemm")
    if prof is not None:
        e1.record()
        side = M * N * out.element_size() * ((aux is not None) + (aux_out is not None) + (epilogue == _lib.EPI_ACCUM))
        prof.append((e0, e1, 2.0 * M * N * K, (M, N, K, bool(a_kmajor), bool(b_kmajor)),
                     float(2 * (M * K + N * K) + M * N * out.element_size() + side)))
    return out


def gemm_grouped2(problems, K, *, a_kmajor=True, b_kmajor=True):
    """Two products in one launch through ptj_gemm_grouped2. problems: two dicts with a, b, out (float32 or bf16 [M, N]), lda,
    ldb, and optionally accumulate, split_k, workspace. Returns False (nothing launched) when the library says the
    pair does not qualify; the caller then issues two gemm() calls."""
    descs = []
    for pr in problems:
        a, b, out = pr["a"], pr["b"], pr["out"]
        if a.dtype != torch.bfloat16 or b.dtype != torch.bfloat16 or out.dtype not in (torch.float32, torch.bfloat16):
            return False
        M, N = out.shape
        split = int(pr.get("split_k", 1))
        ws = pr.get("workspace")
        if split > 1 and (ws is None or ws.numel() < split * M * N):
            ws = torch.empty(split * M * N, device=a.device, dtype=torch.float32)
            pr["workspace"] = ws
        descs.append(_lib.GemmProblem(_ptr(a), _ptr(b), _ptr(out), M, N, pr["lda"], pr["ldb"], out.stride(0), _dt(out),
                                      _lib.EPI_ACCUM if pr.get("accumulate") else _lib.EPI_NONE, split, _ptr(ws),
                                      0 if ws is None else ws.numel()))
    prof = GEMM_PROFILE
    if prof is not None:
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
    rc = _lib.lib().ptj_gemm_grouped2(ctypes.byref(descs[0]), ctypes.byref(descs[1]), K, int(a_kmajor), int(b_kmajor),
                                      _stream())
    if rc == -6:  # PTJ_ERR_UNSUPPORTED: not a pair the thread-block-pair kernel takes
        return False
    _lib.check(rc, "ptj_gemm_grouped2")
    if prof is not None:
        e1.record()
        flops = sum(2.0 * d.M * d.N * K for d in descs)
        nbytes = sum(float(2 * (d.M * K + d.N * K) + d.M * d.N * (2 if d.out_dtype == _lib.PTJ_BF16 else 4)) for d in descs)
        prof.append((e0, e1, flops, ("grouped", descs[0].M, descs[0].N, descs[1].M, descs[1].N, K), nbytes))
    return True


def t_matmul_t(a: torch.Tensor, b: torch.Tensor) -> torch.Tensor:
    """a[N,K] @ b[K,M] (model_triton.py:373-398). No tile-divisibility restrictions."""
    a, b = _cuda(a, "a"), _cuda(b, "b")
    assert a.shape[1] == b.shape[0]
    return gemm(a, b, a_kmajor=True, b_kmajor=False)


def t_linear_fwd_t(layer_params, x: torch.Tensor, activation=None) -> torch.Tensor:
    """x @ W^T + b with W stored [out, in], optional fused tanh-GELU (the linear variant of t_matmul_k,
    model_triton.py:314-321, 364-368; math t_linear_fwd :306-307)."""
    w, bias = _cuda(layer_params[0], "weight"), _f32(layer_params[1])
    x2 = _cuda(x, "x").reshape(-1, x.shape[-1])
    out = gemm(x2, w, bias=bias, epilogue=_lib.EPI_GELU if activation == "gelu" else _lib.EPI_NONE)
    return out.reshape(*x.shape[:-1], w.shape[0])


def t_tlayer_ffn_fwd_t(layer_params, x: torch.Tensor, activation_fn=None) -> torch.Tensor:
    """W2 gelu(W1 x + b1) + b2 with the GELU fused into the first GEMM's epilogue (model_triton.py:1258-1313)."""
    h = t_linear_fwd_t((layer_params[0], layer_params[1]), x, activation="gelu")
    return t_linear_fwd_t((layer_params[2], layer_params[3]), h)


# ---- attention ------------------------------------------------------------------------------------------------------
def _attn_shape(B, H, N, D, q, k, v, o_strides):
    sq, sk, sv = q.stride(), k.stride(), v.stride()
    assert sq[3] == sk[3] == sv[3] == 1, "d_head must be contiguous"
    return AttnShape(B, H, N, D, sq[:3], sk[:3], sv[:3], tuple(o_strides))


def attn_keep_bits(q, k, v, out, seed, stream_id=0, p=None, bits=None):
    """Dropout keep flags of one attention call, to be passed to attn_fwd and attn_bwd (`keep_bits=`) so that the mask
    is drawn once instead of in each kernel. Returns None when the call would not take the tensor-core path or when
    there is nothing to drop. `bits`: optional int32 tensor to reuse."""
    B, H, N, D = q.shape
    p = DROPOUT_RATE if p is None else p
    if p <= 0.0:
        return None
    sh = _attn_shape(B, H, N, D, q, k, v, out.stride()[:3])
    need = int(_lib.lib().ptj_attn_keep_bits_bytes(ctypes.byref(sh), _dt(q)))
    if need == 0:
        return None
    if bits is None or bits.numel() * bits.element_size() < need:
        bits = q.new_empty(need // 4, dtype=torch.int32)
    _lib.check(_lib.lib().ptj_attn_keep_bits(_ptr(bits), ctypes.byref(sh), p, _seed(seed), stream_id, _dt(q), _stream()),
               "ptj_attn_keep_bits")
    return bits


def attn_fwd(q, k, v, out, train, seed, stream_id=0, p=None, keep_bits=None, row_kstart=None):
    """q,k,v,out: [B,H,N,D] strided views (D contiguous). Returns (row_max, row_sum) float32 [B,H,N].
    row_kstart: optional int32 [B,N], first key each query row attends to (see row_kstart_from_mask)."""
    B, H, N, D = q.shape
    row_kstart = _check_kstart(row_kstart, B, N, q.device)
    m = q.new_empty((B, H, N), dtype=torch.float32)
    l = torch.empty_like(m)
    sh = _attn_shape(B, H, N, D, q, k, v, out.stride()[:3])
    p = DROPOUT_RATE if p is None else p
    _lib.check(_lib.lib().ptj_attn_fwd(_ptr(q), _ptr(k), _ptr(v), _ptr(out), _ptr(m), _ptr(l), ctypes.byref(sh), p,
                                       int(bool(train)), _seed(seed), stream_id, _ptr(keep_bits), _ptr(row_kstart), _dt(q),
                                       _stream()),
               "ptj_attn_fwd")
    return m, l


_ATTN_WORKSPACE = {}  # (device, stream) -> byte tensor, grown on demand


def attn_bwd_workspace(nbytes, device):
    """A reusable scratch buffer for attn_bwd on the current stream (contents never carry over between calls)."""
    key = (device, torch.cuda.current_stream(device).cuda_stream)
    buf = _ATTN_WORKSPACE.get(key)
    if buf is None or buf.numel() < nbytes:
        buf = torch.empty(max(nbytes, 16), device=device, dtype=torch.uint8)
        _ATTN_WORKSPACE[key] = buf
    return buf


def attn_bwd(d_o, q, k, v, o, m, l, dq, dk, dv, train, seed, stream_id=0, p=None, workspace=None, keep_bits=None,
             row_kstart=None):
    """workspace: optional uint8 tensor of at least ptj_attn_bwd_workspace_bytes; by default one buffer per
    (device, stream) is kept and reused. row_kstart: the array the forward call was given."""
    B, H, N, D = q.shape
    row_kstart = _check_kstart(row_kstart, B, N, q.device)
    assert d_o.stride() == o.stride(), "dO and O must share a layout"
    sh = _attn_shape(B, H, N, D, q, k, v, o.stride()[:3])
    dsh = _attn_shape(B, H, N, D, dq, dk, dv, o.stride()[:3])
    p = DROPOUT_RATE if p is None else p
    need = int(_lib.lib().ptj_attn_bwd_workspace_bytes(ctypes.byref(sh), _dt(q)))
    if workspace is None and need > 0:
        try:
            workspace = attn_bwd_workspace(need, q.device)
        except torch.OutOfMemoryError:
            if D == 64 and N % 128 == 0:  # (bf16 probabilities: no other kernel rounds them)
                raise
            workspace = None  # the general kernels need none
    wptr = _ptr(workspace) if workspace is not None else None
    wbytes = workspace.numel() * workspace.element_size() if workspace is not None else 0
    _lib.check(
        _lib.lib().ptj_attn_bwd(_ptr(d_o), _ptr(q), _ptr(k), _ptr(v), _ptr(o), _ptr(m), _ptr(l), _ptr(dq), _ptr(dk),
                                _ptr(dv), ctypes.byref(sh), ctypes.byref(dsh), p, int(bool(train)), _seed(seed),
                                stream_id, _ptr(keep_bits), _ptr(row_kstart), wptr, wbytes, _dt(q), _stream()),
        "ptj_attn_bwd")


def _check_kstart(row_kstart, B, N, device):
    if row_kstart is None:
        return None
    if not row_kstart.is_cuda or row_kstart.dtype != torch.int32 or tuple(row_kstart.shape) != (B, N):
        raise ValueError(f"row_kstart must be a CUDA int32 tensor of shape [{B}, {N}]")
    return row_kstart.contiguous()


# Dense masks are checked against the interval form the kernels work with (one host synchronisation per new mask);
# callers that build their masks the way the reference's collator does may switch the check off.
VERIFY_MASKS = True
_KSTART_CACHE = []  # (weak reference to a mask tensor, its version counter, row_kstart): the most recent masks


def row_kstart_from_lengths(doc_lengths, seq: int, device="cuda") -> torch.Tensor:
    """int32 [B, seq] for packed rows: doc_lengths[b] lists the lengths of the documents packed into row b, in order
    (the x_lens / y_lens of the reference's collator, tokenized_dataset.py:206-232); positions beyond their sum are
    padding and attend nothing. Token t of a document that starts at s gets row_kstart = s."""
    out = torch.empty((len(doc_lengths), seq), dtype=torch.int32)
    for b, lens in enumerate(doc_lengths):
        pos = 0
        for n in lens:
            n = min(int(n), seq - pos)
            out[b, pos:pos + n] = pos
            pos += n
        out[b, pos:] = torch.arange(pos, seq, dtype=torch.int32) + 1  # padding: empty range
    return out.to(device)


def row_kstart_from_mask(mask: torch.Tensor) -> torch.Tensor:
    """The kernels' form of a dense attention mask [B, N, N] (True = attend) as the reference's collator builds it:
    causal x block-diagonal over the documents packed into a row x padding (tokenized_dataset.py:110-131). Every row
    of such a mask is an interval of keys that ends at the row's own position (or is empty, for padding rows), so
    the mask is fully described by row_kstart[b, i] = first attended key (i + 1 for an empty row). A mask that is not
    of this form is refused (the check costs one host synchronisation; VERIFY_MASKS = False skips it)."""
    if mask.dim() != 3 or mask.shape[1] != mask.shape[2]:
        raise ValueError("mask must be [B, N, N]")
    # the same tensor object, unmodified since (one batch's mask is used by every layer, forward and backward)
    for ref, version, ks in _KSTART_CACHE:
        if ref() is mask and version == mask._version:
            return ks
    mb = _cuda(mask, "mask").bool()
    B, N, _ = mb.shape
    idx = torch.arange(N, device=mb.device, dtype=torch.int32)
    first = torch.argmax(mb.to(torch.uint8), dim=2).to(torch.int32)  # first True of a row (0 when the row has none)
    kstart = torch.where(mb.any(dim=2), first, idx.view(1, N) + 1)
    if VERIFY_MASKS:
        j = idx.view(1, 1, N)
        rebuilt = (j >= kstart.view(B, N, 1)) & (j <= idx.view(1, N, 1))
        if not torch.equal(rebuilt, mb):
            raise ValueError("attention mask is not causal x block-diagonal x padding: every row must attend an "
                             "interval of keys that ends at its own position (or nothing)")
    _KSTART_CACHE[:] = [e for e in _KSTART_CACHE if e[0]() is not None][-7:]
    _KSTART_CACHE.append((weakref.ref(mask), mask._version, kstart))
    return kstart


def _kstart_or_none(mask):
    """None for no mask or the plain causal one (the fast path), else its row_kstart."""
    if mask is None:
        return None
    ks = row_kstart_from_mask(mask)
    return ks if bool((ks != 0).any()) else None


def t_scaled_dot_prod_attn_fwd3_t(qkv: torch.Tensor, mask: torch.Tensor = None, train=True, p_gen_aux=None):
    """Masked attention on qkv[B,H,3,N,D] -> (out[B,H,N,D], [row_max, row_sum, out]) (model_triton.py:706-754).
    `mask` [B,N,N] bool is applied like the reference kernel applies it (:678-681): it must be causal, optionally
    times the block-diagonal document mask and the padding mask of the reference's collator; None = causal."""
    qkv = _cuda(qkv, "qkv")
    q, k, v = qkv.unbind(dim=2)
    out = qkv.new_empty(q.shape, dtype=qkv.dtype)
    m, l = attn_fwd(q, k, v, out, train, p_gen_aux, row_kstart=_kstart_or_none(mask))
    return out, [m, l, out]


def t_scaled_dot_prod_attn_bkwd3_t(dloss_dx, acts, qkv: torch.Tensor, mask: torch.Tensor = None, train=True,
                                   p_gen_aux=None):
    """(dq, dk, dv), each [B,H,N,D] (model_triton.py:951-1003). Deterministic: no atomics, no zero-filled outputs."""
    qkv = _cuda(qkv, "qkv")
    q, k, v = qkv.unbind(dim=2)
    m, l, out = acts
    d_o = _cuda(dloss_dx, "dloss_dx").to(qkv.dtype).reshape(out.shape)
    out = _cuda(out)
    dq, dk, dv = (qkv.new_empty(q.shape, dtype=qkv.dtype) for _ in range(3))
    attn_bwd(d_o, q, k, v, out, _cuda(m), _cuda(l), dq, dk, dv, train, p_gen_aux, row_kstart=_kstart_or_none(mask))
    return dq, dk, dv


# ---- cross entropy -----------------------------------------------------------------------------------------------------
def cross_entropy(labels, logits, cols=None, want_grad=True, in_place=False, n_valid=None, want_rows=False):
    """Fused CE forward(+backward). logits [rows, ld]; returns (stats float[3] = loss, accuracy, valid fraction;
    n_valid float[1]; dlogits or None), plus the per-row losses float[rows] (0 on padding rows) when want_rows."""
    ld = logits.shape[-1]
    cols = ld if cols is None else cols
    rows = logits.numel() // ld
    labels = _cuda(labels, "labels").reshape(-1).to(torch.int32)
    row_stats = logits.new_empty(2 * rows, dtype=torch.float32)
    out3 = logits.new_empty(3, dtype=torch.float32)
    count = n_valid is None
    if count:
        n_valid = logits.new_empty(1, dtype=torch.float32)
    dlogits = None
    if want_grad:
        dlogits = logits if in_place else torch.empty_like(logits)
    _lib.check(
        _lib.lib().ptj_cross_entropy(_ptr(labels), _ptr(logits), _ptr(dlogits), _ptr(row_stats), _ptr(n_valid),
                                     int(count), _ptr(out3), rows, cols, ld, _dt(logits), _stream()),
        "ptj_cross_entropy")
    if want_rows:
        return out3, n_valid, dlogits, row_stats[:rows]
    return out3, n_valid, dlogits


DECODE_GROUPS = (8, 4, 2, 1)  # sequences in one launch of ptj_decode: the first that its shared memory holds


def decode_greedy(w, cfg, batch: int, start: int, p=None):
    """int32 [batch, cfg.seq]: greedy decoding of `batch` sequences from the token `start` (columns 1.. are written), for
    float32 weights; None where ptj_decode does not apply (other types, sizes or alignments, or tensors that are not what
    the configuration says: the kernel reads them by the configuration's sizes). w: gpt2.Weights."""
    device = w["w_emb"].device
    if any(w[n].dtype != torch.float32 or w[n].data_ptr() % 16 or w[n].device != device or not w[n].is_contiguous()
           or w[n].numel() != math.prod(shape) for n, shape in cfg.param_shapes()) or cfg.seq < 2 or batch < 1:
        return None
    lib, p = _lib.lib(), DROPOUT_RATE if p is None else p
    dims = (cfg.vocab, cfg.dim, cfg.layers, cfg.heads, cfg.ffn, cfg.seq)
    for group in (min(batch, g) for g in DECODE_GROUPS):
        need = int(lib.ptj_decode_workspace_floats(group, *dims))
        if need:
            break
    else:
        return None
    names = [n for n, _ in cfg.param_shapes() if n.startswith("l")]
    ptrs = torch.tensor([w[n].data_ptr() for n in names], dtype=torch.int64, device=device)
    tokens = torch.empty((batch, cfg.seq), device=device, dtype=torch.int32)
    ws = torch.empty(need, device=device, dtype=torch.float32)
    for b0 in range(0, batch, group):
        n = min(batch - b0, group)
        _lib.check(lib.ptj_decode(_ptr(w["w_emb"]), _ptr(w["b_head"]), _ptr(w["w_pos"]), _ptr(ptrs), _ptr(w["g_f"]),
                                  _ptr(w["b_f"]), _ptr(tokens[b0:]), start, p, n, *dims, _ptr(ws), ws.numel(), _stream()),
                   "ptj_decode")
    return tokens


def argmax_rows(x: torch.Tensor, cols=None) -> torch.Tensor:
    """int32[rows] = index of the largest of the first `cols` elements of every row of x [rows, ld] (first index on
    ties): the torch.argmax of the reference's greedy decoding loop (loss_and_optimizer_triton.py:207)."""
    if not x.is_cuda:
        raise RuntimeError("x must live on a CUDA device: there is no CPU implementation")
    assert x.dim() == 2 and x.stride(1) == 1, "rows may be strided, elements of a row must be contiguous"
    rows, ld = x.shape[0], x.stride(0)
    cols = x.shape[1] if cols is None else cols
    out = x.new_empty(rows, dtype=torch.int32)
    _lib.check(_lib.lib().ptj_argmax_rows(_ptr(x), _ptr(out), rows, cols, ld, _dt(x), _stream()), "ptj_argmax_rows")
    return out


def t_avg_cross_entropy_loss(y_labels: torch.Tensor, x_logits: torch.Tensor):
    """(mean loss over labels != 0, number of such labels) (loss_and_optimizer_triton.py:23-32)."""
    out3, n_valid, _ = cross_entropy(y_labels, _cuda(x_logits, "x_logits"), want_grad=False)
    return out3[0], n_valid[0].to(torch.int64)


def t_avg_cross_entropy_loss_bkwd3_t(y_labels: torch.Tensor, x_logits: torch.Tensor):
    """(loss[1], n_valid, dlogits) (loss_and_optimizer_triton.py:176-197)."""
    x = _cuda(x_logits, "x_logits")
    out3, n_valid, dlogits = cross_entropy(y_labels, x, want_grad=True)
    return out3[0:1], n_valid[0].to(torch.int64), dlogits.reshape(x_logits.shape)


def accuracy_from_logits(y_labels: torch.Tensor, x_logits: torch.Tensor):
    """Mean over labels != 0 of argmax == label (loss_and_optimizer_triton.py:199-200), from the same kernel."""
    out3, _, _ = cross_entropy(y_labels, _cuda(x_logits, "x_logits"), want_grad=False)
    return out3[1]


# ---- embedding ------------------------------------------------------------------------------------------------------
def embed_fwd(ids, w_emb, w_pos, train, seed, stream_id=0, out_dtype=None, p=None):
    """dropout(w_emb[ids] * sqrt(D) + w_pos) -> [B, S, D] (model_triton.py:166-167, 2338-2341)."""
    B, S = ids.shape
    V, D = w_emb.shape
    ids = _cuda(ids, "ids").to(torch.int32)
    out_dtype = out_dtype or w_emb.dtype
    y = w_emb.new_empty((B, S, D), dtype=out_dtype)
    p = DROPOUT_RATE if p is None else p
    _lib.check(
        _lib.lib().ptj_embed_fwd(_ptr(ids), _ptr(w_emb), _ptr(w_pos), _ptr(y), B, S, D, V, p, int(bool(train)),
                                 _seed(seed), stream_id, _dt(w_emb), _dt(y), _stream()), "ptj_embed_fwd")
    return y


def embed_bwd(dy, ids, d_w_emb, d_w_pos, accumulate, train, seed, stream_id=0, sorted_pos=None, p=None):
    """Scatter the (dropout-masked) gradient into d_w_emb [V,D] (optionally accumulating) and d_w_pos [S,D]."""
    B, S = ids.shape
    V, D = d_w_emb.shape
    ids = _cuda(ids, "ids").to(torch.int32)
    if sorted_pos is None:
        sorted_pos = torch.sort(ids.reshape(-1), stable=True).indices.to(torch.int32)
    p = DROPOUT_RATE if p is None else p
    _lib.check(
        _lib.lib().ptj_embed_bwd(_ptr(dy), _ptr(ids), _ptr(sorted_pos), _ptr(d_w_emb), _ptr(d_w_pos), int(accumulate), B,
                                 S, D, V, p, int(bool(train)), _seed(seed), stream_id, _dt(dy), _stream()),
        "ptj_embed_bwd")


def colsum(x2d, cols=None, out=None):
    """Column sums of a [rows, ld] matrix (first `cols` columns) in float32: bias gradients."""
    rows, ld = x2d.shape
    cols = ld if cols is None else cols
    if out is None:
        out = x2d.new_empty(cols, dtype=torch.float32)
    n = _lib.lib().ptj_colsum_scratch_floats(rows, cols)
    scratch = x2d.new_empty(max(n, 1), dtype=torch.float32)
    _lib.check(_lib.lib().ptj_colsum(_ptr(x2d), _ptr(out), _ptr(scratch), n, rows, cols, ld, _dt(x2d), _stream()),
               "ptj_colsum")
    return out


def gelu_bwd_colsum(dy2d, x_preact2d, colsum_out=None, in_place=False):
    """(dy * gelu'(x_preact), its column sums in float32) in one pass over [rows, cols] matrices: the FFN's hidden
    gradient and the gradient of its first bias (model_triton.py:296-304 followed by the db of :423-434)."""
    dy, x = _cuda(dy2d, "dy"), _cuda(x_preact2d, "x_preact")
    assert dy.dim() == 2 and dy.shape == x.shape and dy.dtype == x.dtype
    rows, cols = dy.shape
    dx = dy if in_place else torch.empty_like(dy)
    out = colsum_out if colsum_out is not None else dy.new_empty(cols, dtype=torch.float32)
    n = _lib.lib().ptj_colsum_scratch_floats(rows, cols)
    scratch = dy.new_empty(max(n, 1), dtype=torch.float32)
    _lib.check(_lib.lib().ptj_gelu_bwd_colsum(_ptr(dy), _ptr(x), _ptr(dx), _ptr(out), _ptr(scratch), n, rows, cols, cols,
                                              _dt(dy), _stream()), "ptj_gelu_bwd_colsum")
    return dx, out


def last_kernel_fault() -> int:
    code = ctypes.c_uint(0)
    _lib.check(_lib.lib().ptj_last_kernel_fault(_stream(), ctypes.byref(code)), "ptj_last_kernel_fault")
    return int(code.value)

