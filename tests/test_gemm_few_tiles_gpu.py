"""PTJ_SPLIT_TAIL on products of fewer 256 x 256 tiles than half of the thread-block pairs: all rows split over K."""
import pytest
import torch

from conftest import pkg
from oracle import philox

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,parts", [(3072, 768, 3072, 2), (513, 776, 2056, 8), (256, 256, 2048, 8), (2304, 1024, 4096, 2)])
@pytest.mark.parametrize("epilogue", ["none", "dropout"])
def test_all_rows_in_parts(M, N, K, parts, epilogue):
    ops, lib = pkg("operators"), pkg("_lib")
    assert int(lib.lib().ptj_gemm_tail_split_floats(M, N, K)) == parts * M * N
    assert int(lib.lib().ptj_gemm_tail_split_rows(M, N, K)) == 0
    g = torch.Generator(device="cuda").manual_seed(M)
    a, res = (torch.randn(M, n, generator=g, device="cuda").bfloat16() for n in (K, N))
    b = (0.05 * torch.randn(*((N, K) if epilogue == "dropout" else (K, N)), generator=g, device="cuda")).bfloat16()
    bias = torch.randn(N, generator=g, device="cuda")
    if epilogue == "dropout":
        kw = dict(bias=bias, epilogue=lib.EPI_DROPOUT_RESID, aux=res, dropout_args=(0.3, True, 99, 2))
        acc = a.double() @ b.double().t() + bias.double()
        keep = torch.from_numpy(philox.keep_mask(99, 2, M * N, 0.3)).view(M, N).cuda()
        ref = res.double() + acc * keep
    else:
        kw = dict(b_kmajor=False, N=N, K=K, M=M)
        ref = a.double() @ b.double()
    got = ops.gemm(a, b, split_k=ops.SPLIT_TAIL, **kw)
    plain = ops.gemm(a, b, **kw)
    assert ops.last_kernel_fault() == 0
    # one rounding to bf16, and float32 sums of K products of magnitude |a| |b| < 0.05 * 16 or so: 2^-20 of sqrt(K)
    bound = 2.0 ** -8 * ref.abs() + 2.0 ** -20 * K ** 0.5
    assert bool(((got.double() - ref).abs() <= bound).all()) and bool(((plain.double() - ref).abs() <= bound).all())
    again = ops.gemm(a, b, split_k=ops.SPLIT_TAIL, **kw)
    assert torch.equal(got, again)
