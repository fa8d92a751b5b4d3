"""Attention on the tensor cores with float32 probabilities in three bf16 parts (bf16 operands; every row length and head size
but whole tiles of 64-wide heads) against float64: edges of tiles, narrow and wide heads, one to several tiles and items."""
import ctypes
import math

import pytest
import torch

from conftest import pkg
from oracle import philox
from test_attn_general_gpu import documents, reference, run

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B,H,S,D,p,train,packed", [
    (1, 1, 1, 16, 0.1, True, False),       # one row, the narrowest head
    (2, 1, 128, 32, 0.1, True, False),     # one whole tile of half a sub-tile
    (1, 2, 255, 24, 0.1, True, True),
    (1, 1, 257, 64, 0.0, True, False),     # one row in the last tile
    (2, 2, 256, 72, 0.1, True, False),     # eight columns in the second sub-tile
    (1, 2, 385, 96, 0.1, False, False),    # evaluation: probabilities times 1 - p
    (1, 3, 511, 128, 0.1, True, True),     # 511 % 8 == 7: keep flags start inside a call
    (5, 32, 130, 64, 0.1, True, False),    # more items than blocks: several a block, single tiles among them
    (3, 50, 192, 128, 0.1, True, True),
])
def test_against_float64(B, H, S, D, p, train, packed):
    ops = pkg("operators")
    g = torch.Generator(device="cuda").manual_seed(S + D)
    q, k, v, do = (torch.randn(B, H, S, D, generator=g, device="cuda").bfloat16() for _ in range(4))
    ks = ops.row_kstart_from_lengths(documents(B, S, packed), S) if packed else None
    (o, m, l, dq, dk, dv), bufs = run(ops, q, k, v, do, p, train, 99, ks, 0)
    assert all(bool((flat[-512:] == 7.0).all()) for flat in bufs), "a store went beyond the tensor"
    keep = torch.ones((), device="cuda", dtype=torch.float64)
    if train and p > 0:
        keep = torch.from_numpy(philox.keep_mask(99, 0, B * H * S * S, p)).view(B, H, S, S).cuda().double()
    # the bound of the general kernels: one rounding of the result, and 2^-17 of the sum of magnitudes for scores and sums
    refs = reference(q, k, v, do, o, keep, 1.0 if train else 1.0 - p, ks)
    for name, got, (ref, mag) in zip(("O", "dQ", "dK", "dV"), (o, dq, dk, dv), refs):
        worst = ((got.double() - ref).abs() - 2.0 ** -8 * ref.abs() - 2.0 ** -17 * mag).max()
        assert bool(torch.isfinite(got.float()).all()) and float(worst) <= 1e-30, f"{name} {float(worst):.3e}"


@pytest.mark.parametrize("S,D", [(500, 64), (131, 32), (256, 128)])
def test_keep_flags_and_a_missing_workspace(S, D):
    """Flags drawn beforehand give what the kernels draw themselves; a backward call without a workspace (the general
    kernels then) gives the same up to one rounding of the result."""
    ops = pkg("operators")
    B, H, p, seed = 2, 3, 0.2, 11
    g = torch.Generator(device="cuda").manual_seed(S)
    q, k, v, do = (torch.randn(B, H, S, D, generator=g, device="cuda").bfloat16() for _ in range(4))
    res = []
    for how in ("kernel", "flags", "no workspace"):
        o, dq, dk, dv = (torch.empty_like(q) for _ in range(4))
        bits = ops.attn_keep_bits(q, k, v, o, seed, p=p) if how == "flags" else None
        assert (bits is not None) == (how == "flags")
        m, l = ops.attn_fwd(q, k, v, o, True, seed, p=p, keep_bits=bits)
        ops.attn_bwd(do, q, k, v, o, m, l, dq, dk, dv, True, seed, p=p, keep_bits=bits,
                     workspace=torch.empty(0, device="cuda", dtype=torch.uint8) if how == "no workspace" else None)
        res.append((o, m, l, dq, dk, dv))
    torch.cuda.synchronize()
    assert ops.last_kernel_fault() == 0
    assert all(torch.equal(a, b) for a, b in zip(res[0], res[1]))
    # two roundings to bf16 of values that differ by float32 errors: at most one unit in the last place (2^-7 of the value)
    for a, b in zip(res[0], res[2]):
        assert bool(((a.double() - b.double()).abs() <= 2.0 ** -7 * b.double().abs() + 1e-5).all())


@pytest.mark.parametrize("S,D,p,flags,packed", [
    (300, 128, 0.1, False, False),  # single buffers, three tiles: operands are looked at after the tile before is done
    (300, 128, 0.1, True, True),
    (500, 64, 0.2, True, False),    # four tiles, two groups, flags drawn beforehand
    (260, 32, 0.0, False, True),
])
@pytest.mark.parametrize("what", ["one", "rows", "all"])
def test_nonfinite_operands_give_what_the_general_kernels_give(S, D, p, flags, packed, what):
    """Infinities and NaNs in Q, K, V or dO over several tiles: the same elements of every result are infinite or NaN as from
    the general kernels, which rows on an odd stride run on, and the others agree."""
    ops = pkg("operators")
    B, H, seed = 3, 60, 5  # several items a block: what one meets does not reach the next
    g = torch.Generator(device="cuda").manual_seed(S + D)
    clean = [torch.randn(B, H, S, D, generator=g, device="cuda").bfloat16() for _ in range(4)]
    ks = ops.row_kstart_from_lengths(documents(B, S, packed), S) if packed else None
    bad = torch.tensor([math.nan, math.inf, -math.inf], device="cuda").bfloat16()
    spread = lambda t: torch.nn.functional.pad(t, (0, 3))[..., :D]
    for which in range(4):
        x = [t.clone() for t in clean]
        if what == "one":
            x[which][0, 1, S // 2, D // 2] = bad[1]
            x[which][1, 5, S - 3, 1] = bad[0]
            x[which][2, 59, 0, D - 1] = bad[2]
        elif what == "rows":
            x[which][:, ::3, 5:S:37] = bad[torch.randint(0, 3, (B, H // 3, len(range(5, S, 37)), D), generator=g, device="cuda")]
        else:
            x[which][:, ::2] = bad[0]
        q, k, v, do = x
        o, dq, dk, dv = (torch.empty_like(q) for _ in range(4))
        bits = ops.attn_keep_bits(q, k, v, o, seed, p=p) if flags else None
        assert (bits is not None) == flags
        m, l = ops.attn_fwd(q, k, v, o, True, seed, p=p, keep_bits=bits, row_kstart=ks)
        ops.attn_bwd(do, q, k, v, o, m, l, dq, dk, dv, True, seed, p=p, keep_bits=bits, row_kstart=ks)
        sq, sk, sv, sdo, so, go, gq, gk, gv = (spread(t) for t in (q, k, v, do, o, o, dq, dk, dv))
        gm, _ = ops.attn_fwd(sq, sk, sv, go, True, seed, p=p, row_kstart=ks)
        ops.attn_bwd(sdo, sq, sk, sv, so, m, l, gq, gk, gv, True, seed, p=p, row_kstart=ks)
        torch.cuda.synchronize()
        assert ops.last_kernel_fault() == 0
        for name, got, want in (("O", o, go), ("maximum", m, gm), ("dQ", dq, gq), ("dK", dk, gk), ("dV", dv, gv)):
            got, want = got.double(), want.double()
            same = torch.where(torch.isfinite(want), torch.isfinite(got), (got == want) | (got.isnan() & want.isnan()))
            assert bool(same.all()), (which, name, int((~same).sum()))
            # two roundings to bf16, 2^-8 of the value each, and 2^-17 of sums of magnitudes (below 32) for float32 sums
            err = (got - want).abs()[torch.isfinite(want)] - 2.0 ** -7 * want.abs()[torch.isfinite(want)]
            assert err.numel() == 0 or float(err.max()) <= 2.0 ** -12, (which, name, float(err.max()))


@pytest.mark.parametrize("S,D", [(300, 128), (200, 64)])
def test_statistics_of_rows_whose_scores_are_all_minus_infinity(S, D):
    """The maximum is -inf then, and the sum of exponentials 0, as from the general kernels."""
    ops = pkg("operators")
    q = torch.ones(1, 2, S, D, device="cuda", dtype=torch.bfloat16)
    k, v = torch.full_like(q, 0.5), torch.ones_like(q)
    k[:, :, :40, 3] = -math.inf  # rows up to 39 attend nothing else
    o = torch.empty_like(q)
    m, l = ops.attn_fwd(q, k, v, o, True, 1, p=0.0)
    assert bool((m[..., :40] == -math.inf).all()) and bool((l[..., :40] == 0).all()) and bool(o[:, :, :40].isnan().all())
    rows = torch.arange(1, S - 39, device="cuda", dtype=torch.float32)  # equal scores
    assert bool(torch.isfinite(m[..., 40:]).all()) and bool(((l[..., 40:] - rows).abs() <= 2.0 ** -20 * rows).all())


def test_beyond_four_gigabytes_of_shares_the_general_kernels_run():
    """dQ shares grow with the square of the row length: from 4 GiB on the call asks for no workspace, and each half of the
    batch, which has its shares, gives the same up to two roundings."""
    ops, lib = pkg("operators"), pkg("_lib")
    B, H, S, D = 2, 64, 8065, 32
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, do = (torch.randn(B, H, S, D, generator=g, device="cuda").bfloat16() for _ in range(4))

    def workspace(n):
        sh = lib.AttnShape(n, H, S, D, *[q.stride()[:3]] * 4)
        return lib.lib().ptj_attn_bwd_workspace_bytes(ctypes.byref(sh), lib.PTJ_BF16)

    assert workspace(2) == 0 and 2 ** 31 < workspace(1) < 2 ** 32
    o, *whole = (torch.empty_like(q) for _ in range(4))
    m, l = ops.attn_fwd(q, k, v, o, True, 1, p=0.0)
    ops.attn_bwd(do, q, k, v, o, m, l, *whole, True, 1, p=0.0)
    halves = [torch.empty_like(q) for _ in range(3)]
    for b in range(2):
        one = lambda t: t[b:b + 1]
        ops.attn_bwd(*map(one, (do, q, k, v, o, m, l, *halves)), True, 1, p=0.0)
    torch.cuda.synchronize()
    ops._ATTN_WORKSPACE.clear()
    assert ops.last_kernel_fault() == 0
    for name, a, b in zip(("dQ", "dK", "dV"), whole, halves):
        # two roundings to bf16, and 2^-17 of sums of magnitudes (below 64) for float32 sums of up to 8065 terms
        err = ((a.double() - b.double()).abs() - 2.0 ** -7 * a.double().abs()).max()
        assert float(err) <= 2.0 ** -11, (name, float(err))
