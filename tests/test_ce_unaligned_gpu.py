"""bf16 cross entropy on rows that start anywhere (odd vocabulary without padding) against float64."""
import math

import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,cols,shift", [(9, 1, 0), (9, 5, 3), (17, 13, 0), (64, 1003, 1), (5, 4099, 7), (450, 8193, 5)])
def test_rows_of_any_phase(rows, cols, shift):
    ops = pkg("operators")
    g = torch.Generator().manual_seed(rows + cols)
    flat = torch.randn(rows * cols + shift, generator=g).mul_(4).bfloat16().cuda()
    x = flat[shift:].view(rows, cols)
    labels = torch.randint(0, cols, (rows,), generator=g).to(torch.int32).cuda()
    buf = torch.full((rows * cols + shift + 64,), 7.0, device="cuda", dtype=torch.bfloat16)
    grad = buf[shift:shift + rows * cols].view(rows, cols)  # same phase as the logits
    grad.copy_(x)
    stats, n, d = ops.cross_entropy(labels, grad, want_grad=True, in_place=True)
    xd, valid = x.double(), labels > 0
    if not bool(valid.any()):
        return
    lp = torch.log_softmax(xd, dim=1)
    nv = valid.sum()
    loss = -(lp.gather(1, labels.long()[:, None]).squeeze(1) * valid).sum() / nv
    ref = (lp.exp() - torch.nn.functional.one_hot(labels.long(), cols)) * valid[:, None] / nv
    assert abs(float(stats[0]) - float(loss)) <= 1e-5 * max(1.0, abs(float(loss)))
    assert float(stats[1]) == pytest.approx(float(((xd.argmax(1) == labels) & valid).sum() / nv))
    # bf16 result: half an ulp of 2^-8, and 2^-18 of the exponential's argument (|x - max| < 40)
    assert bool(((d.double() - ref).abs() <= 2.0 ** -8 * ref.abs() + 1e-9).all())
    assert bool((buf[shift + rows * cols:] == 7.0).all()) and bool((buf[:shift] == 7.0).all())


@pytest.mark.parametrize("cols,shift", [(1003, 1), (515, 0)])
def test_rows_of_large_magnitude(cols, shift):
    """The shift by the row's maximum is exact, whatever its size: rows around 10^4, where the product with log2(e) rounded
    to float32 errs by 2^-11, and rows that hold the type's lowest value, where it overflows."""
    ops = pkg("operators")
    lowest = torch.finfo(torch.bfloat16).min
    rows = torch.full((6, cols), -20000.0)
    rows[0, 2:5] = 10048.0                        # three equal maxima
    rows[1] = -10048.0                            # all equal
    rows[2] = lowest                              # everything masked
    rows[3], rows[3, 5] = lowest, 3.0             # one entry left
    rows[4], rows[4, 5], rows[4, 7] = -math.inf, 3.0, 3.0
    rows[5] = 30000.0 + 128.0 * torch.arange(cols).remainder(3)
    flat = torch.zeros(6 * cols + shift, device="cuda", dtype=torch.bfloat16)
    x = flat[shift:].view(6, cols)
    x.copy_(rows)
    labels = torch.tensor([3, 9, 1, 5, 7, 2], dtype=torch.int32, device="cuda")
    grad = torch.empty_like(flat)[shift:].view(6, cols)
    grad.copy_(x)
    _, _, d, loss = ops.cross_entropy(labels, grad, want_grad=True, in_place=True, want_rows=True)
    lp = torch.log_softmax(x.double(), dim=1)
    ref = -lp.gather(1, labels.long()[:, None]).squeeze(1)
    # float32: a logarithm and a sum of equal powers of two of at most 1003 terms
    assert float((loss.double() - ref).abs().max()) <= 2e-6, (loss, ref)
    want = (lp.exp() - torch.nn.functional.one_hot(labels.long(), cols)) / 6
    assert bool(((d.double() - want).abs() <= 2.0 ** -8 * want.abs() + 2e-7).all())
