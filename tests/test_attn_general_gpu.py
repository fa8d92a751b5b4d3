"""The general attention kernels (float32 arithmetic for every shape, stride and type that the tensor-core kernels do not
take) against float64: several tiles in both directions, dropout, packed documents, any head size and any row stride."""
import math

import pytest
import torch

from conftest import pkg
from oracle import philox

pytestmark = pytest.mark.gpu
GUARD = 512  # elements behind every output that must keep their value
BF16, F32 = torch.bfloat16, torch.float32


def guarded(shape, dtype, stride_pad):
    """An output tensor (rows `stride_pad` elements apart from the next) and the guard elements behind it."""
    B, H, S, D = shape
    n = B * H * S * (D + stride_pad)
    flat = torch.full((n + GUARD,), 7.0, device="cuda", dtype=dtype)
    return flat[:n].view(B, H, S, D + stride_pad)[..., :D], flat


def run(ops, q, k, v, do, p, train, seed, ks, pad):
    """Forward and backward of one call: outputs, and the buffers behind O, dQ, dK, dV."""
    shape, dtype = tuple(q.shape), q.dtype
    (o, fo), (dq, fq), (dk, fk), (dv, fv) = (guarded(shape, dtype, pad) for _ in range(4))
    spread = lambda t: torch.nn.functional.pad(t, (0, pad))[..., :shape[-1]] if pad else t
    q, k, v, do = (spread(t) for t in (q, k, v, do))
    m, l = ops.attn_fwd(q, k, v, o, train, seed, p=p, row_kstart=ks)
    ops.attn_bwd(do, q, k, v, o, m, l, dq, dk, dv, train, seed, p=p, row_kstart=ks)
    torch.cuda.synchronize()
    assert ops.last_kernel_fault() == 0
    return (o, m, l, dq, dk, dv), (fo, fq, fk, fv)


def reference(q, k, v, do, o_got, keep, eval_scale, ks):
    """(value, sum of magnitudes) of O, dQ, dK, dV in float64. delta is formed from the output as the kernel rounded it."""
    q, k, v, do, o_got = (t.double() for t in (q, k, v, do, o_got))
    S, scale = q.shape[2], 1.0 / math.sqrt(q.shape[3])
    i = torch.arange(S, device="cuda")
    on = (i.view(1, 1, S) <= i.view(1, S, 1)) & (i.view(1, 1, S) >= (ks.view(-1, S, 1) if ks is not None else 0))
    on = on.unsqueeze(1)
    s = (q @ k.transpose(-1, -2) * scale).masked_fill(~on, -math.inf)
    some = on.any(dim=-1, keepdim=True)
    p = torch.softmax(s.masked_fill(~some, 0.0), dim=-1) * on
    f = keep * eval_scale
    dp, delta = do @ v.transpose(-1, -2), (do * o_got).sum(-1, keepdim=True)
    ds, ds_abs = p * (dp * f - delta) * scale, p * ((dp * f).abs() + (do * o_got).abs().sum(-1, keepdim=True)) * scale
    t = lambda x: x.transpose(-1, -2)
    return [((p * f) @ v, (p * f) @ v.abs()), (ds @ k, ds_abs @ k.abs()), (t(ds) @ q, t(ds_abs) @ q.abs()),
            (t(p * f) @ do, t(p * f) @ do.abs())]


def documents(B, S, packed):
    return [[max(1, S // 3), S // 2]] * (B - 1) + [[1, max(1, S - 2)]] if packed else None


@pytest.mark.parametrize("dtype,B,H,S,D,p,train,packed,pad", [
    # bf16 shapes that fill no tensor-core tile
    (BF16, 1, 1, 1, 64, 0.1, True, False, 0),      # a single row
    (BF16, 2, 3, 7, 32, 0.1, True, True, 0),
    (BF16, 1, 2, 127, 64, 0.1, True, False, 0),
    (BF16, 1, 2, 129, 64, 0.0, True, True, 0),
    (BF16, 4, 3, 500, 64, 0.1, True, False, 0),    # 500 % 8 == 4: flags start anywhere in a byte
    (BF16, 2, 2, 500, 64, 0.1, True, True, 0),
    (BF16, 2, 2, 384, 32, 0.1, True, False, 0),    # whole tensor-core tiles along the sequence, half of one along the head
    (BF16, 1, 5, 641, 8, 0.1, False, False, 0),    # smallest head, evaluation scaling
    (BF16, 2, 2, 200, 128, 0.1, True, True, 0),
    (BF16, 2, 2, 256, 64, 0.2, True, True, 3),     # whole tiles, but rows on odd strides
    # float32: several tiles with dropout and documents, every head instantiation, heads that are no multiple of four
    (F32, 2, 2, 200, 64, 0.2, True, True, 0),
    (F32, 1, 3, 333, 32, 0.2, True, False, 0),     # odd rows: the flag phase moves from row to row and tile to tile
    (F32, 2, 2, 333, 80, 0.2, True, True, 0),
    (F32, 1, 2, 200, 128, 0.2, True, True, 0),
    (F32, 1, 2, 130, 127, 0.1, True, False, 0),
    (F32, 2, 1, 193, 65, 0.0, True, True, 0),
    (F32, 2, 2, 129, 33, 0.2, True, True, 3),      # rows on odd strides
    (F32, 2, 1, 257, 64, 0.1, False, True, 1),
])
def test_against_float64(dtype, B, H, S, D, p, train, packed, pad):
    ops = pkg("operators")
    g = torch.Generator(device="cuda").manual_seed(S + D)
    q, k, v, do = (torch.randn(B, H, S, D, generator=g, device="cuda").to(dtype) for _ in range(4))
    lens = documents(B, S, packed)
    ks = ops.row_kstart_from_lengths(lens, S) if packed else None
    (o, m, l, dq, dk, dv), bufs = run(ops, q, k, v, do, p, train, 99, ks, pad)
    for flat in bufs:
        assert bool((flat[-GUARD:] == 7.0).all()), "a store went beyond the tensor"
        if pad:
            assert bool((flat[:-GUARD].view(-1, D + pad)[:, D:] == 7.0).all()), "a store went between the rows"
    keep = torch.ones((), device="cuda", dtype=torch.float64)
    if train and p > 0:
        keep = torch.from_numpy(philox.keep_mask(99, 0, B * H * S * S, p)).view(B, H, S, S).cuda().double()
    refs = reference(q, k, v, do, o, keep, 1.0 if train else 1.0 - p, ks)
    # Only the result is rounded to the output type (2^-8 of it in bf16, 2^-24 in float32). The rest is float32: scores of
    # at most 128 terms err by some 2^-24 of |q| |k| / sqrt(D) < 30, which shifts a probability by as much relatively, and
    # the sums over up to 641 keys by less; 2^-17 of the sum of magnitudes covers both. A probability rounded to bf16
    # would err by 2^-8 of the largest terms of that sum.
    u = 2.0 ** -8 if dtype == BF16 else 2.0 ** -24
    for name, got, (ref, mag) in zip(("O", "dQ", "dK", "dV"), (o, dq, dk, dv), refs):
        worst = ((got.double() - ref).abs() - u * ref.abs() - 2.0 ** -17 * mag).max()
        assert bool(torch.isfinite(got.float()).all()) and float(worst) <= 1e-30, f"{name} {float(worst):.3e}"


@pytest.mark.parametrize("bad", [math.nan, math.inf, -math.inf])
@pytest.mark.parametrize("dtype,S,D,p,packed", [(F32, 200, 64, 0.0, False), (F32, 200, 32, 0.2, True), (F32, 130, 80, 0.0, True),
                                                (BF16, 150, 64, 0.1, True)])
def test_nonfinite_rows_reach_only_what_attends_them(dtype, S, D, p, packed, bad):
    """A NaN or an infinity in one row of V, K, Q or dO must not reach an output whose mask leaves that row out, although
    both lie in the same tile: those outputs are bit for bit what they are without it."""
    ops = pkg("operators")
    B, H, row = 1, 2, S - 40  # inside the last tile but one of the sequence, and of a document
    lens = [[max(1, S // 3), S - S // 3 - 20]] if packed else None
    ks = ops.row_kstart_from_lengths(lens, S) if packed else None
    g = torch.Generator(device="cuda").manual_seed(S)
    clean = [torch.randn(B, H, S, D, generator=g, device="cuda").to(dtype) for _ in range(4)]
    first = ks[0].long() if packed else torch.zeros(S, dtype=torch.long, device="cuda")
    i = torch.arange(S, device="cuda")
    attends = (row >= first) & (row <= i)        # query rows that read key `row`
    attended = (i >= first[row]) & (i <= row)    # keys that query row `row` reads
    want, _ = run(ops, *clean, p, True, 7, ks, 0)
    for which in range(4):
        x = [t.clone() for t in clean]
        x[which][0, 1, row, D // 2] = bad
        (o, m, l, dq, dk, dv), _ = run(ops, *x, p, True, 7, ks, 0)
        own = i == row
        queries = {0: own, 1: attends, 2: attends, 3: own}[which]  # rows of O and dQ that may change
        keys = attended
        if which in (1, 2):  # every key of a row that attends `row` shares its normalisation and its delta
            keys = torch.zeros_like(own)
            for r in i[attends].tolist():
                keys |= (i >= first[r]) & (i <= r)
        for name, got, ref, may in (("O", o, want[0], queries if which != 3 else ~own & own), ("dQ", dq, want[3], queries),
                                    ("dK", dk, want[4], keys), ("dV", dv, want[5], keys)):
            assert torch.equal(got[:, 0], ref[:, 0]), (which, name, "another head")
            same = got[0, 1][~may] == ref[0, 1][~may]
            assert bool(same.all()), (which, name, int((~same).any(dim=1).sum()))
        if which == 2:  # and it does reach the rows that attend it
            assert not bool(torch.isfinite(o[0, 1, row]).all())
