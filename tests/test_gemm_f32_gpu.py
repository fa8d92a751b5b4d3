"""float32 products on the tensor cores (operands split into three bf16 parts) against float64, and next to the
fused-multiply-add kernel that runs the same product when no workspace is given."""
import ctypes

import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ops():
    return pkg("operators")


def launches(fn):
    lib = pkg("_lib")
    before = lib.launch_count()
    fn()
    return lib.launch_count() - before


def operand(rows, cols, ld, seed, kmajor):
    g = torch.Generator(device="cuda").manual_seed(seed)
    # magnitudes over several powers of two, so that all three parts of an element matter
    x = torch.randn(rows, cols, generator=g, device="cuda") * torch.exp2(4 * torch.rand(rows, cols, generator=g, device="cuda"))
    store = torch.zeros((rows, ld) if kmajor else (cols, ld), device="cuda")
    if kmajor:
        store[:, :cols] = x
    else:
        store[:, :rows] = x.t()
    return x, store


def bound(K, absum):
    """Chains of 64 products: four truncating additions at full magnitude (2^-23 each), smaller partial products and what
    the split leaves out below 2^-24; the chains are added with rounding (2^-24 each). All relative to sum |a b|."""
    return (9.0 + K / 64.0) * 2.0 ** -24 * absum


@pytest.mark.parametrize("a_k,b_k", [(True, True), (True, False), (False, True), (False, False)])
@pytest.mark.parametrize("M,N,K,pad", [(256, 256, 256, 0), (257, 300, 333, 3), (1000, 2000, 72, 1), (64, 1500, 4097, 4),
                                       (520, 776, 768, 0)])
def test_layouts_edges_and_k_split(ops, a_k, b_k, M, N, K, pad):
    A, sa = operand(M, K, (K if a_k else M) + pad, 1, a_k)
    B, sb = operand(N, K, (K if b_k else N) + pad, 2, b_k)
    ref = A.double() @ B.double().t()
    absum = A.double().abs() @ B.double().abs().t()
    out = torch.full((M, N), float("nan"), device="cuda")
    n = launches(lambda: ops.gemm(sa, sb, a_kmajor=a_k, b_kmajor=b_k, M=M, N=N, K=K, lda=sa.shape[1], ldb=sb.shape[1], out=out))
    assert n >= 2  # the splitting pass and the product (and the sum of K parts): not the one-launch FMA kernel
    assert bool(((out.double() - ref).abs() <= bound(K, absum)).all())
    fma = torch.empty_like(out)
    lib = pkg("_lib")
    lib.check(lib.lib().ptj_gemm(sa.data_ptr(), sb.data_ptr(), fma.data_ptr(), 0, 0, 0, M, N, K, sa.shape[1], sb.shape[1],
                                 N, int(a_k), int(b_k), 0, 0, 0, None, 1, 0, 0, torch.cuda.current_stream().cuda_stream), "ptj_gemm")
    rms = lambda x: float((x.double() - ref).pow(2).mean().sqrt())
    print("rms error / rms value: tensor cores %.2e, FMA %.2e" % (rms(out) / float(ref.pow(2).mean().sqrt()), rms(fma) / float(ref.pow(2).mean().sqrt())))
    assert rms(out) <= rms(fma)  # measured: 0.7 of it at K = 72, 0.1 at K = 4096
    again = torch.empty_like(out)
    ops.gemm(sa, sb, a_kmajor=a_k, b_kmajor=b_k, M=M, N=N, K=K, lda=sa.shape[1], ldb=sb.shape[1], out=again)
    assert torch.equal(out, again)
    assert ops.last_kernel_fault() == 0


@pytest.mark.parametrize("M,N,K", [(512, 768, 3072), (300, 264, 256), (300, 261, 1000)])
def test_epilogues_match_the_fma_kernel(ops, M, N, K):
    """Bias, GELU with the saved pre-activation, GELU', dropout + residual and accumulation, with and without parts of K."""
    lib = pkg("_lib")
    A, B = torch.randn(M, K, device="cuda") / K ** 0.5, torch.randn(N, K, device="cuda")
    bias, aux = torch.randn(N, device="cuda"), torch.randn(M, N, device="cuda")
    for mode, kw in ((lib.EPI_NONE, dict(bias=bias)), (lib.EPI_GELU, dict(bias=bias, aux_out=True)), (lib.EPI_GELU_BWD, dict(aux=aux)),
                     (lib.EPI_DROPOUT_RESID, dict(bias=bias, aux=aux)), (lib.EPI_ACCUM, {})):
        got, ref = [], []
        for dst, ws_floats in ((got, 1), (ref, 0)):
            out = aux.clone()
            pre = torch.empty(M, N, device="cuda") if kw.get("aux_out") else None
            need = lib.lib().ptj_gemm_f32_workspace_floats(M, N, K, 1, 1) * ws_floats
            ws = torch.empty(max(need, 4), device="cuda")
            drop = ctypes.byref(lib.DropoutArgs(0.1, 1, 1234, 0)) if mode == lib.EPI_DROPOUT_RESID else None
            ptr = lambda t: 0 if t is None else t.data_ptr()
            lib.check(lib.lib().ptj_gemm(A.data_ptr(), B.data_ptr(), out.data_ptr(), ptr(kw.get("bias")), ptr(kw.get("aux")),
                                         ptr(pre), M, N, K, K, K, N, 1, 1, 0, 0, mode, drop, 1, ws.data_ptr() if need else 0,
                                         need, torch.cuda.current_stream().cuda_stream), "ptj_gemm")
            dst += [out] + ([pre] if pre is not None else [])
        for a, b in zip(got, ref):
            # both are within a few float32 roundings of the exact product (values of size one)
            assert float((a - b).abs().max()) <= 2e-5


def test_extreme_values(ops):
    """The largest finite float32 (by fused multiply-adds), a small number's last bit and zeros come through; a NaN stays where
    it belongs."""
    M = N = 256
    A, B = torch.zeros(M, 256, device="cuda"), torch.zeros(N, 256, device="cuda")
    A[0, 0], B[0, 0] = torch.finfo(torch.float32).max, 1.0
    A[1, 1], B[1, 1] = 1e-30, 1.0 + 2.0 ** -23
    A[2, 2], B[2, 2] = float("nan"), 1.0
    out = ops.gemm(A, B)
    assert float(out[0, 0]) == torch.finfo(torch.float32).max
    assert abs(float(out[1, 1]) / 1e-30 - 1.0) < 3e-7
    assert bool(torch.isnan(out[2]).all()) and not bool(torch.isnan(out[[0, 1, 3]]).any())


def fma_product(ops, sa, sb, M, N, K, a_k, b_k):
    """The same product on the fused-multiply-add kernel: no workspace."""
    lib, out = pkg("_lib"), torch.empty(M, N, device="cuda")
    lib.check(lib.lib().ptj_gemm(sa.data_ptr(), sb.data_ptr(), out.data_ptr(), 0, 0, 0, M, N, K, sa.shape[1], sb.shape[1],
                                 N, int(a_k), int(b_k), 0, 0, 0, None, 1, 0, 0, torch.cuda.current_stream().cuda_stream), "ptj_gemm")
    return out


@pytest.mark.parametrize("a_k,b_k,M,N,K", [(True, True, 300, 520, 256), (True, False, 257, 333, 700), (False, True, 64, 130, 4200),
                                           (False, False, 520, 776, 768)])
def test_infinite_and_huge_operands_match_the_fma_kernel(ops, a_k, b_k, M, N, K):
    """An infinity gives the infinities (and the NaNs of inf - inf and inf * 0) that it gives in a float32 sum, and products
    that overflow do so where a float32 sum does; both bit for bit as on the fused-multiply-add kernel."""
    g = torch.Generator(device="cuda").manual_seed(M + K)
    base = [torch.randn(r, K, generator=g, device="cuda") for r in (M, N)]
    for case in ("inf in A", "-inf in B", "both", "huge", "overflow"):
        A, B = (t.clone() for t in base)
        if case in ("inf in A", "both"):
            A[3, 5] = A[M - 1, K - 1] = float("inf")
            B[7, 5] = 0.0
        if case in ("-inf in B", "both"):
            B[N - 1, 5] = -float("inf")
        if case == "huge":
            A[2] *= 2.0 ** 100
            B[4] *= 2.0 ** -100
        if case == "overflow":
            A[1] *= 2.0 ** 120
            B[9] *= 2.0 ** 30
        sa, sb = A if a_k else A.t().contiguous(), B if b_k else B.t().contiguous()
        kw = dict(a_kmajor=a_k, b_kmajor=b_k, M=M, N=N, K=K, lda=sa.shape[1], ldb=sb.shape[1])
        got, want = ops.gemm(sa, sb, **kw), fma_product(ops, sa, sb, M, N, K, a_k, b_k)
        assert torch.equal(torch.isnan(got), torch.isnan(want)), case
        assert torch.equal(torch.nan_to_num(got, nan=0.0), torch.nan_to_num(want, nan=0.0)), case
        if case == "inf in A":
            assert bool(torch.isinf(got[3]).sum() == N - 1) and bool(torch.isnan(got[3, 7]))
        # the epilogue runs on what the sum gave: accumulation, bias and GELU
        lib, bias = pkg("_lib"), torch.randn(N, generator=g, device="cuda")
        acc, pre = torch.ones(M, N, device="cuda"), torch.empty(M, N, device="cuda")
        ops.gemm(sa, sb, **kw, out=acc, epilogue=lib.EPI_ACCUM)
        assert torch.equal(torch.nan_to_num(acc, nan=0.0), torch.nan_to_num(want + 1.0, nan=0.0)), case
        ops.gemm(sa, sb, **kw, bias=bias, epilogue=lib.EPI_GELU, aux_out=pre)
        assert torch.equal(torch.nan_to_num(pre, nan=0.0), torch.nan_to_num(want + bias, nan=0.0)), case
    assert ops.last_kernel_fault() == 0


@pytest.mark.parametrize("ea,eb", [(-120, 0), (-140, 10), (-126, 20), (0, -133), (-70, -60)])
@pytest.mark.parametrize("a_k,b_k,K", [(True, True, 300), (False, False, 2100)])
def test_small_magnitudes_keep_all_their_bits(ops, a_k, b_k, K, ea, eb):
    """Operands down to float32's subnormals: their last bits lie far below bf16's smallest value."""
    M, N = 264, 300
    g = torch.Generator(device="cuda").manual_seed(K)
    A, B = (torch.ldexp(1.0 + torch.rand(r, K, generator=g, device="cuda"), torch.tensor(e, device="cuda"))
            * (torch.randint(0, 2, (r, K), generator=g, device="cuda") * 2 - 1) for r, e in ((M, ea), (N, eb)))
    sa, sb = A if a_k else A.t().contiguous(), B if b_k else B.t().contiguous()
    out = ops.gemm(sa, sb, a_kmajor=a_k, b_kmajor=b_k, M=M, N=N, K=K, lda=sa.shape[1], ldb=sb.shape[1])
    ref, absum = A.double() @ B.double().t(), A.double().abs() @ B.double().abs().t()
    # results below 2^-126 are rounded to multiples of 2^-149, once per chain and part of K at most
    assert bool(((out.double() - ref).abs() <= bound(K, absum) + (K / 64 + 8) * 2.0 ** -149).all())
