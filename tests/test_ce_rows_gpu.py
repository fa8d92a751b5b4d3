"""The bf16 cross entropy that holds a row in registers, against float64: a few columns around the widths at which the threads
per row change and at which the three-pass kernel takes over, more rows than blocks, padding rows among them, in place."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [2, 9, 255, 2047, 14335, 14336, 14337, 28673, 57344, 57345])
@pytest.mark.parametrize("pad", [0, 3])  # rows one after the other (any phase), rows padded to a multiple of eight
def test_against_float64(cols, pad):
    ops = pkg("operators")
    rows = 700 if cols < 3000 else 160  # more than the resident blocks of either form
    ld = (cols + 7) // 8 * 8 if pad else cols
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = (2.0 * torch.randn(rows, ld, generator=g, device="cuda")).bfloat16()
    y = torch.randint(1, cols, (rows,), generator=g, device="cuda", dtype=torch.int32)
    y[::5] = 0                                        # padding labels: no contribution, zero gradient
    x[1, cols - 1], y[1] = 40.0, cols - 1             # the label is the maximum, in the row's last column
    x[2, 0] = x[2, y[2].item()] = 41.0                # a tie whose first index is not the label
    ref = x[:, :cols].double()
    on = y > 0
    lse = torch.logsumexp(ref, 1)
    picked = ref.gather(1, y.long().view(-1, 1)).squeeze(1)
    n = int(on.sum())
    want = torch.softmax(ref, 1)
    want[torch.arange(rows, device="cuda"), y.long()] -= 1.0
    want = want * on.view(-1, 1) / n
    col = torch.arange(cols, device="cuda").expand(rows, cols)
    first = col.masked_fill(ref != ref.amax(1, keepdim=True), cols).amin(1)  # the first column that holds the maximum
    hits = int(((first == y) & on).sum())
    buf = torch.cat([x.reshape(-1), x.new_full((64,), 7.0)])
    stats, n_valid, d = ops.cross_entropy(y, buf[:rows * ld].view(rows, ld), cols=cols, want_grad=True, in_place=True)
    assert bool((buf[-64:] == 7.0).all()), "a store went beyond the rows"
    assert int(n_valid) == n and abs(float(stats[1]) * n - hits) < 0.5
    # float32 exponentials and sums of up to 57345 terms: some 2^-20 of the loss
    assert abs(float(stats[0]) - float((lse - picked)[on].sum() / n)) <= 2.0 ** -20 * float(lse.abs().max())
    # one rounding to bf16 (2^-9), and 2^-16 of 1 / n where the label's element cancels
    err = (d[:, :cols].double() - want).abs() - 2.0 ** -8 * want.abs() - 2.0 ** -16 / n
    assert float(err.max()) <= 0.0
    if pad and ld > cols:
        assert torch.equal(d[:, cols:], x[:, cols:]), "padding columns keep their values"
