"""The bf16 cross entropy that holds a row in registers or in shared memory, against float64: a few columns around the widths at
which the threads per row change and at which the other kernels take over, several rows a block, padding rows among them, in place
and without a gradient."""
import threading

import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [2, 9, 255, 2047, 14335, 14336, 14337, 20001, 28673, 50257, 57344, 57345])
@pytest.mark.parametrize("pad", [0, 3])  # rows one after the other (any phase), rows padded to a multiple of eight
def test_against_float64(cols, pad):
    ops = pkg("operators")
    rows = 1300  # at least two for each of the 592, 444 or 296 blocks; odd columns one after the other: of another phase
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
    loss = float((lse - picked)[on].sum() / n)
    buf = torch.cat([x.reshape(-1), x.new_full((64,), 7.0)])
    alone, _, _ = ops.cross_entropy(y, buf[:rows * ld].view(rows, ld), cols=cols, want_grad=False)
    stats, n_valid, d = ops.cross_entropy(y, buf[:rows * ld].view(rows, ld), cols=cols, want_grad=True, in_place=True)
    assert bool((buf[-64:] == 7.0).all()), "a store went beyond the rows"
    assert int(n_valid) == n and abs(float(stats[1]) * n - hits) < 0.5
    # float32 exponentials and sums of up to 57345 terms: some 2^-20 of the loss
    assert abs(float(stats[0]) - loss) <= 2.0 ** -20 * float(lse.abs().max())
    assert torch.equal(alone, stats), "the same sums whether a gradient follows or not"
    # one rounding to bf16 (2^-9), and 2^-16 of 1 / n where the label's element cancels
    err = (d[:, :cols].double() - want).abs() - 2.0 ** -8 * want.abs() - 2.0 ** -16 / n
    assert float(err.max()) <= 0.0
    if pad and ld > cols:
        assert torch.equal(d[:, cols:], x[:, cols:]), "padding columns keep their values"


@pytest.mark.parametrize("cols", [20001, 50257])  # held in registers, held in shared memory
def test_bits_do_not_depend_on_where_a_row_is_held(cols):
    """Every kernel adds up a row in the same order, the elements behind its last whole vector last: a row padded with -inf to
    the width of the kernel that reads rows three times, its last element moved to that row's end, gives the same bits."""
    ops = pkg("operators")
    rows, wide, ld = 4096, 57345, 57352
    g = torch.Generator(device="cuda").manual_seed(cols)
    x = (2.0 * torch.randn(rows, (cols + 7) // 8 * 8, generator=g, device="cuda")).bfloat16()
    x[:, [0, 1, 2, 3, 4, 5, 6, 7, 4096, 4097, cols - 1]] += 10.0  # elements of one thread that decide the sum
    y = torch.randint(1, cols - 1, (rows,), generator=g, device="cuda", dtype=torch.int32)
    z = torch.full((rows, ld), -float("inf"), device="cuda", dtype=torch.bfloat16)
    z[:, :cols - 1] = x[:, :cols - 1]
    z[:, wide - 1] = x[:, cols - 1]
    _, _, d, loss = ops.cross_entropy(y, x, cols=cols, want_grad=True, want_rows=True)
    _, _, e, want = ops.cross_entropy(y, z, cols=wide, want_grad=True, want_rows=True)
    assert torch.equal(loss, want)
    assert torch.equal(d[:, :cols - 1], e[:, :cols - 1]) and torch.equal(d[:, cols - 1], e[:, wide - 1])


def test_vocabularies_of_several_threads():
    """The shared memory that a kernel may use is a property of the kernel, not of a launch: a narrow call on one thread must
    not lower it under a wide one on another."""
    lib, failed, together = pkg("_lib").lib(), [], threading.Barrier(6)

    def work(cols):
        x = torch.zeros(1, cols, device="cuda", dtype=torch.bfloat16)
        y = torch.ones(1, device="cuda", dtype=torch.int32)
        out, n = torch.empty(5, device="cuda"), torch.ones(1, device="cuda")
        stream = torch.cuda.Stream()
        torch.cuda.synchronize()
        args = (y.data_ptr(), x.data_ptr(), None, out.data_ptr(), n.data_ptr(), 0, out.data_ptr() + 8, 1, cols, cols,
                pkg("_lib").PTJ_BF16, stream.cuda_stream)
        together.wait()
        for _ in range(2000):
            rc = lib.ptj_cross_entropy(*args)
            if rc != 0:
                failed.append((cols, rc))
                return

    threads = [threading.Thread(target=work, args=(cols,)) for cols in (57344, 30000) * 3]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    assert not failed
