"""bf16 cross entropy on rows that start anywhere (odd vocabulary without padding) against float64."""
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
