"""Tensor-core attention at row lengths and head sizes that fill no tile (rows and columns beyond the tensor are zeros in
the tiles and must reach no output), against the general kernels, which views with an odd row stride are routed to."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu
TOL = 2e-2   # P and dS are rounded to bf16 (2^-9 each) before they are multiplied
GUARD = 512  # elements behind every output that must keep their value


def err(a, b):
    """max |a - b| on the scale of the reference or of the unit-variance inputs, whichever is larger: a row with a single
    key has dS = P (dP - delta) = 0, where both kernels leave the rounding of the two 64-term float32 sums (< 64 * 2^-24
    of their terms)."""
    a, b = a.double(), b.double()
    return float((a - b).abs().max()) / max(1.0, float(b.abs().max()))


def guarded(*shape):
    n = 1
    for s in shape:
        n *= s
    flat = torch.full((n + GUARD,), 7.0, device="cuda", dtype=torch.bfloat16)
    return flat[:n].view(*shape), flat[n:]


def odd_rows(t):
    """The same values with a row stride that no vector load or tensor map takes."""
    return torch.nn.functional.pad(t, (0, 3))[..., :t.shape[-1]]


def run(ops, q, k, v, do, outs, seed, train, bits, ks):
    o, dq, dk, dv = outs
    keep = ops.attn_keep_bits(q, k, v, o, seed) if bits and train else None
    m, l = ops.attn_fwd(q, k, v, o, train, seed, keep_bits=keep, row_kstart=ks)
    ops.attn_bwd(do, q, k, v, o, m, l, dq, dk, dv, train, seed, keep_bits=keep, row_kstart=ks)
    return o, m, l, dq, dk, dv


@pytest.mark.parametrize("B,H,S,D,p,train,packed", [
    (1, 1, 1, 64, 0.1, True, False),      # a single row
    (2, 3, 7, 32, 0.1, True, True),       # odd rows: mask words start anywhere in a call
    (1, 2, 127, 64, 0.1, True, False),
    (1, 2, 129, 64, 0.0, True, True),     # one row in the second tile
    (4, 3, 500, 64, 0.1, True, False),    # 500 % 8 == 4
    (2, 2, 500, 64, 0.1, True, True),
    (2, 2, 384, 32, 0.1, True, False),    # whole tiles along the sequence, half of one along the head
    (1, 5, 641, 8, 0.1, False, False),    # smallest head, evaluation scaling
    (8, 40, 136, 56, 0.1, True, True),    # more items than thread blocks
])
def test_ragged_matches_general_kernels(B, H, S, D, p, train, packed):
    ops = pkg("operators")
    g = torch.Generator(device="cuda").manual_seed(S + D)
    q, k, v, do = (torch.randn(B, H, S, D, generator=g, device="cuda").bfloat16() for _ in range(4))
    ks = None
    if packed:
        ks = ops.row_kstart_from_lengths([[max(1, S // 3), S // 2] for _ in range(B)], S)
    ops.DROPOUT_RATE = p
    try:
        ref = run(ops, *(odd_rows(t) for t in (q, k, v, do)),
                  [odd_rows(torch.empty(B, H, S, D, device="cuda", dtype=torch.bfloat16)) for _ in range(4)],
                  99, train, False, ks)
        for bits in (False, True):
            outs, tails = zip(*(guarded(B, H, S, D) for _ in range(4)))
            got = run(ops, q, k, v, do, outs, 99, train, bits, ks)
            torch.cuda.synchronize()
            assert ops.last_kernel_fault() == 0
            assert all(bool((t == 7.0).all()) for t in tails), "a store went beyond the tensor"
            for name, a, b in zip(("O", "max", "sum", "dQ", "dK", "dV"), got, ref):
                assert bool(torch.isfinite(a.float()).all()), name
                assert err(a, b) < TOL, f"{name} {err(a, b):.3e}"
    finally:
        ops.DROPOUT_RATE = 0.1
