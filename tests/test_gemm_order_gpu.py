"""bf16 products whose A operand does not fit the L2 take their tiles in another order: the same bits as the product of its rows in
blocks that do, whose tiles are the same."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("a_kmajor,b_kmajor,out_dtype,N,split", [
    (True, True, torch.bfloat16, 700, 1), (True, False, torch.bfloat16, 768, 1), (False, False, torch.float32, 700, 1),
    (False, False, torch.float32, 520, 2)])
def test_bits_do_not_depend_on_the_order_of_tiles(a_kmajor, b_kmajor, out_dtype, N, split):
    ops = pkg("operators")
    M, K, cut = 33000, 2048, 65 * 256  # A: 135 MB, its two blocks 68 and 67; the last row of tiles is ragged
    g = torch.Generator(device="cuda").manual_seed(N)
    a = torch.randn(*((M, K) if a_kmajor else (K, M)), generator=g, device="cuda").bfloat16()
    b = torch.randn(*((N, K) if b_kmajor else (K, (N + 7) // 8 * 8)), generator=g, device="cuda").bfloat16()
    guard = torch.full((M + 1, N), 7.0, device="cuda", dtype=out_dtype)

    def product(a, rows, out):
        ops.gemm(a, b, a_kmajor=a_kmajor, b_kmajor=b_kmajor, M=rows, N=N, K=K, lda=a.stride(0), ldb=b.stride(0), out=out, split_k=split)

    product(a, M, guard[:M])
    parts = torch.empty(M, N, device="cuda", dtype=out_dtype)
    for m0, m1 in ((0, cut), (cut, M)):
        product(a[m0:m1] if a_kmajor else a[:, m0:m1], m1 - m0, parts[m0:m1])
    torch.cuda.synchronize()
    assert ops.last_kernel_fault() == 0
    assert torch.equal(guard[:M], parts) and bool((guard[M] == 7.0).all())
    rows = torch.arange(0, M, 997, device="cuda")
    want = (a[rows] if a_kmajor else a[:, rows].t()).double() @ (b.t() if b_kmajor else b[:, :N]).double()
    # one rounding of the result (2^-8 in bf16), and float32 sums of 2048 products of rms 1, some 45 together
    u = 2.0 ** -8 if out_dtype == torch.bfloat16 else 2.0 ** -24
    assert bool(((guard[rows].double() - want).abs() <= u * want.abs() + 2.0 ** -9).all())
