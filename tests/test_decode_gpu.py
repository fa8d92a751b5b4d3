"""Greedy decoding with kept keys and values against the same loop over whole forward passes, at sizes that fill no chunk,
part, block share or lane group of the kernel, and the alignments that its entry point takes."""
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
    (5, 300, 1280, 3, 20, 5120, 10),  # rows of which shared memory holds four: groups of four and one
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
    # every sequence starts alike, so all are equal: a mix-up between sequences could not show, to a caller neither
    assert torch.equal(ids, ids[:1].expand_as(ids))
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


def decode_from(params, cfg, B, start, vectors, w_qkv_offset=0):
    """ptj_decode with every vector `vectors` floats and the first layer's W_QKV `w_qkv_offset` floats off a 16-byte boundary."""
    lib, ops, gpt2 = pkg("_lib"), pkg("operators"), pkg("gpt2")
    w = gpt2.Weights.from_pytree(params, cfg, torch.float32)
    moved = {}
    for n, t in w.t.items():
        off = vectors if t.dim() == 1 else (w_qkv_offset if n == "l0.w_qkv" else 0)
        buf = torch.zeros(t.numel() + 4, device="cuda")
        buf[off:off + t.numel()] = t.reshape(-1)
        moved[n] = buf[off:off + t.numel()]
        assert moved[n].data_ptr() % 16 == 4 * off
    ptrs = torch.tensor([moved[n].data_ptr() for n, _ in cfg.param_shapes() if n.startswith("l")], dtype=torch.int64, device="cuda")
    dims = (cfg.vocab, cfg.dim, cfg.layers, cfg.heads, cfg.ffn, cfg.seq)
    ws = torch.empty(lib.lib().ptj_decode_workspace_floats(B, *dims), device="cuda")
    tokens = torch.full((B, cfg.seq), -7, device="cuda", dtype=torch.int32)
    m = {n: t.data_ptr() for n, t in moved.items()}
    rc = lib.lib().ptj_decode(m["w_emb"], m["b_head"], m["w_pos"], ptrs.data_ptr(), m["g_f"], m["b_f"], tokens.data_ptr(), start,
                              ops.DROPOUT_RATE, B, *dims, ws.data_ptr(), ws.numel(), torch.cuda.current_stream().cuda_stream)
    return rc, ops.last_kernel_fault(), tokens


@pytest.mark.parametrize("offset", [1, 2, 3])
def test_vectors_on_any_float(offset):
    ops, gpt2 = pkg("operators"), pkg("gpt2")
    params = weights(1001, 96, 2, 3, 388, 33, 5)
    cfg = gpt2.config_from_params(params, ops.DROPOUT_RATE)
    rc, fault, tokens = decode_from(params, cfg, 2, 1000, offset)
    assert (rc, fault) == (0, 0)
    want = ops.decode_greedy(gpt2.Weights.from_pytree(params, cfg, torch.float32), cfg, 2, 1000)
    assert torch.equal(tokens[:, 1:], want[:, 1:]) and want[0, 1:].unique().numel() > 2


def test_a_misaligned_matrix_is_reported():
    ops, gpt2 = pkg("operators"), pkg("gpt2")
    params = weights(64, 32, 1, 2, 64, 8, 3)
    cfg = gpt2.config_from_params(params, ops.DROPOUT_RATE)
    rc, fault, tokens = decode_from(params, cfg, 1, 1, 0, w_qkv_offset=1)
    assert (rc, fault) == (0, 0x3102) and bool((tokens == -7).all())
    assert decode_from(params, cfg, 1, 1, 0)[:2] == (0, 0)
