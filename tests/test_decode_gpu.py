"""Greedy decoding with kept keys and values against the same loop over whole forward passes, at sizes that fill no chunk,
part, block share or lane group of the kernel."""
import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


def weights(V, D, L, H, F, S, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = lambda *s, sd=1.0: torch.randn(*s, generator=g, device="cuda") * sd
    # residual branches that outweigh the token embedding: at the scale of fresh weights the tied head repeats its input
    layer = lambda: [1 + n(D, sd=0.02), n(D, sd=0.02), n(H, 3, D // H, D, sd=D ** -0.5), n(D, D, sd=8 * D ** -0.5),
                     1 + n(D, sd=0.02), n(D, sd=0.02), n(F, D, sd=D ** -0.5), n(F, sd=0.02), n(D, F, sd=8 * F ** -0.5),
                     n(D, sd=0.02)]
    return [[n(V, D, sd=0.02), n(V, sd=0.02)], [n(S, D, sd=0.5)]] + [layer() for _ in range(L)] + [[1 + n(D, sd=0.02), n(D, sd=0.02)]]


@pytest.mark.parametrize("B,V,D,L,H,F,S", [
    (1, 17, 8, 1, 2, 4, 2),           # smallest: fewer rows than blocks, one token
    (2, 1001, 96, 2, 3, 388, 33),     # rows shorter than a chunk, odd vocabulary, 4 F no multiple of a chunk
    (3, 5003, 320, 2, 4, 1280, 70),   # 80-wide heads (20 of 32 lanes), more positions than lane groups
    (5, 1024, 256, 1, 4, 1024, 9),    # five sequences in the kernel for eight
    (8, 300, 1024, 1, 8, 4096, 40),   # largest activations: the shallow ring
    (11, 513, 128, 3, 2, 512, 20),    # two groups of sequences
])
def test_decode_matches_whole_forward(B, V, D, L, H, F, S):
    ops, ev, gpt2 = pkg("operators"), pkg("evaluate"), pkg("gpt2")
    params = weights(V, D, L, H, F, S, V + D)
    cfg = gpt2.config_from_params(params, ops.DROPOUT_RATE)
    w = gpt2.Weights.from_pytree(params, cfg, torch.float32)
    start = V - 1
    got = ops.decode_greedy(w, cfg, B, start)
    assert got is not None and ops.last_kernel_fault() == 0
    # teacher-forced: the whole forward over the decoded tokens must rank each of them first. float32 sums of up to 4096
    # terms in another order differ by about 1e-6 of the logits' scale; a token may win only within ten times that.
    ids = got.long()
    ids[:, 0] = start
    assert torch.equal(ids, ids[:1].expand_as(ids))  # every sequence starts alike
    logits = ev.t_gpt2_forward(params, ids[:2], None, None, False).double()
    top = logits[:, :-1].max(dim=-1).values
    mine = logits[:, :-1].gather(2, ids[:2, 1:, None]).squeeze(2)
    assert float((top - mine).max()) <= 1e-5 * float(logits.abs().max())
    if S > 8:
        assert ids[0].unique().numel() > 2, "the check needs a sequence that moves"
    assert ev.predict(params, B, None, S, start, -1).shape == (B, S - 1)


def test_other_weights_take_the_whole_forward():
    ops, gpt2 = pkg("operators"), pkg("gpt2")
    for D, H, F in ((24, 4, 96), (8, 2, 4)):  # 6-wide heads; 8-wide rows in bf16
        params = weights(64, D, 1, H, F, 8, 3)
        dtype = torch.float32 if D == 24 else torch.bfloat16
        cfg = gpt2.config_from_params(params, 0.1)
        assert ops.decode_greedy(gpt2.Weights.from_pytree(params, cfg, dtype), cfg, 2, 1) is None
