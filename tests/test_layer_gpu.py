"""A layer's launches issued by one library call against the same launches issued one by one: the same bits."""
import ctypes
import threading

import pytest
import torch

from conftest import pkg

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,dim,heads,ffn,layers,B,S,p,packed", [
    (torch.bfloat16, 128, 4, 512, 2, 4, 128, 0.0, False),   # 32-wide heads, no dropout: no keep flags
    (torch.bfloat16, 256, 4, 1000, 3, 2, 200, 0.1, True),   # ragged rows, documents, an FFN width that fills no tile
    (torch.bfloat16, 768, 12, 3072, 1, 8, 1024, 0.1, False),  # tail splits, pairs of weight gradients, K parts
    (torch.bfloat16, 64, 1, 192, 0, 1, 64, 0.1, False),     # no layer at all
    (torch.float32, 256, 2, 512, 2, 2, 96, 0.1, True),
    (torch.float32, 40, 5, 72, 1, 3, 17, 0.1, False),       # everything on the general kernels
])
@pytest.mark.parametrize("train", [True, False])
def test_same_bits_as_single_launches(dtype, dim, heads, ffn, layers, B, S, p, packed, train):
    ops, gpt2 = pkg("operators"), pkg("gpt2")
    cfg = gpt2.GPT2Config(vocab=304, dim=dim, layers=layers, heads=heads, ffn=ffn, seq=S, dropout=p)
    g = torch.Generator(device="cuda").manual_seed(1)
    flat = [0.05 * torch.randn(s, generator=g, device="cuda") + (1.0 if gpt2.base_name(n)[0] == "g" else 0.0)
            for n, s in cfg.param_shapes()]
    w = gpt2.Weights.from_pytree(gpt2.unflatten_like(flat, cfg), cfg, dtype)
    y = torch.randint(1, 304, (B, S + 1), generator=g, device="cuda", dtype=torch.int32)
    ks = ops.row_kstart_from_lengths([[max(1, S // 3), S // 2]] * B, S) if packed else None
    seeds = list(range(5, 6 + 3 * layers))
    results = []
    try:
        for single in (False, True):
            ops.GEMM_PROFILE = [] if single else None
            step, ready = gpt2.Gpt2Step(cfg, dtype), []
            grads = {n: torch.full(s, 3.0, device="cuda") for n, s in cfg.param_shapes()}
            stats = step.loss_and_grads(w, grads, y, train, seeds, row_kstart=ks, on_ready=ready.extend)
            results.append([stats] + [grads[n] for n, _ in cfg.param_shapes()])
            assert sorted(ready) == sorted(grads)
            logits, _ = step.forward(w, y[:, :-1].contiguous(), train, seeds, row_kstart=ks)
            results[-1].append(logits[:, :304])
    finally:
        ops.GEMM_PROFILE = None
    assert ops.last_kernel_fault() == 0
    assert all(torch.equal(a, b) for a, b in zip(*results))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_strided_weights_and_gradients(dtype):
    """Matrices that are columns of wider ones: the same bits as contiguous ones, and nothing is written between the rows."""
    ops, gpt2 = pkg("operators"), pkg("gpt2")
    cfg = gpt2.GPT2Config(vocab=304, dim=256, layers=2, heads=4, ffn=512, seq=200, dropout=0.1)
    g = torch.Generator(device="cuda").manual_seed(2)
    flat = [0.05 * torch.randn(s, generator=g, device="cuda") + (1.0 if gpt2.base_name(n)[0] == "g" else 0.0)
            for n, s in cfg.param_shapes()]
    w = gpt2.Weights.from_pytree(gpt2.unflatten_like(flat, cfg), cfg, dtype)
    y = torch.randint(1, 304, (2, 201), generator=g, device="cuda", dtype=torch.int32)
    names = [n for n, s in cfg.param_shapes() if n.startswith("l") and len(s) == 2]  # (W_qkv is used as one matrix)

    def wide(t):
        buf = torch.full((t.shape[0], t.shape[1] + 24), 7.0, device="cuda", dtype=t.dtype)
        buf[:, :t.shape[1]] = t
        return buf, buf[:, :t.shape[1]]

    def step(weights, grads):
        stats = gpt2.Gpt2Step(cfg, dtype).loss_and_grads(gpt2.Weights(cfg, weights), grads, y, True, list(range(5, 12)))
        torch.cuda.synchronize()
        assert ops.last_kernel_fault() == 0
        return [stats] + [grads[n] for n, _ in cfg.param_shapes()]

    def fresh():
        return {n: torch.full(s, 3.0, device="cuda") for n, s in cfg.param_shapes()}

    want = step(w.t, fresh())
    got = step({n: wide(t)[1] if n in names else t for n, t in w.t.items()}, fresh())
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    buffers = {n: wide(t) for n, t in fresh().items() if n in names}
    got = step(w.t, {**fresh(), **{n: view for n, (_, view) in buffers.items()}})
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    assert all(bool((buf[:, view.shape[1]:] == 7.0).all()) for buf, view in buffers.values())


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_one_engine_on_two_streams_and_threads(dtype):
    """Passes of one engine side by side, each on a stream and a thread of its own: the bits of passes one after the other."""
    gpt2 = pkg("gpt2")
    cfg = gpt2.GPT2Config(vocab=304, dim=256, layers=4, heads=4, ffn=1024, seq=256, dropout=0.1)
    g = torch.Generator(device="cuda").manual_seed(3)
    flat = [0.05 * torch.randn(s, generator=g, device="cuda") + (1.0 if gpt2.base_name(n)[0] == "g" else 0.0)
            for n, s in cfg.param_shapes()]
    w = gpt2.Weights.from_pytree(gpt2.unflatten_like(flat, cfg), cfg, dtype)
    ys = [torch.randint(1, 304, (4, 257), generator=g, device="cuda", dtype=torch.int32) for _ in range(2)]
    step = gpt2.Gpt2Step(cfg, dtype)

    def passes(i, out, n):
        for _ in range(n):
            grads = {name: torch.empty(s, device="cuda") for name, s in cfg.param_shapes()}
            stats = step.loss_and_grads(w, grads, ys[i], True, list(range(100 * i, 100 * i + 13)))
            out.append([stats] + list(grads.values()))

    want = [[], []]
    for i in range(2):
        passes(i, want[i], 1)
    torch.cuda.synchronize()
    got, streams = [[], []], [torch.cuda.Stream() for _ in range(2)]

    def work(i):
        with torch.cuda.stream(streams[i]):
            passes(i, got[i], 8)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(2):
        assert len(got[i]) == 8
        assert all(torch.equal(a, b) for one in got[i] for a, b in zip(one, want[i][0]))


@pytest.mark.parametrize("dim,heads,S", [(256, 4, 200), (128, 4, 384)])  # ragged rows; 32-wide heads
def test_a_step_without_room_for_flags_and_workspace(dim, heads, S, monkeypatch):
    """bf16 attention off whole tiles of 64-wide heads needs neither keep flags nor a workspace: a step that finds no room for
    them takes the flags from the kernels and the general backward kernels, and needs no more memory than that."""
    ops, gpt2, lib = pkg("operators"), pkg("gpt2"), pkg("_lib")
    cfg = gpt2.GPT2Config(vocab=304, dim=dim, layers=2, heads=heads, ffn=4 * dim, seq=S, dropout=0.1)
    g = torch.Generator(device="cuda").manual_seed(4)
    flat = [0.05 * torch.randn(s, generator=g, device="cuda") + (1.0 if gpt2.base_name(n)[0] == "g" else 0.0)
            for n, s in cfg.param_shapes()]
    w = gpt2.Weights.from_pytree(gpt2.unflatten_like(flat, cfg), cfg, torch.bfloat16)
    B = 4
    y = torch.randint(1, 304, (B, S + 1), generator=g, device="cuda", dtype=torch.int32)
    plan = gpt2._LayerPlan(cfg, torch.bfloat16, B, S, True, True)
    attention = lib.lib().ptj_attn_bwd_workspace_bytes(
        ctypes.byref(lib.AttnShape(B, heads, S, dim // heads, *[(3 * S * dim, 3 * dim // heads, 3 * dim)] * 3,
                                   (S * dim, dim // heads, dim))), lib.PTJ_BF16)
    assert 0 < 4 * plan.ws_least[1] < attention <= 4 * plan.ws_floats[1] and plan.keep_bytes > 0
    small = gpt2._LayerPlan(cfg, torch.bfloat16, B, S, True, False)
    real, limit = torch.empty, [None]

    def empty(*shape, **kw):
        if limit[0] is not None and shape in limit[0]:
            raise torch.OutOfMemoryError("no room")
        return real(*shape, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    results = []
    for short in (False, True):
        limit[0] = [(plan.act_bytes,), (plan.ws_floats[1],)] if short else None
        step = gpt2.Gpt2Step(cfg, torch.bfloat16)
        grads = {n: torch.zeros(s, device="cuda") for n, s in cfg.param_shapes()}
        stats = step.loss_and_grads(w, grads, y, True, list(range(5, 12)))
        torch.cuda.synchronize()
        assert ops.last_kernel_fault() == 0
        results.append((stats, grads))
        kept = sum(t.numel() for t in step._ws.values())
        assert kept <= max(small.ws_least[1], small.ws_floats[0]) if short else kept >= plan.ws_floats[1]
    (want, a), (got, b) = results
    assert torch.equal(want, got)  # the forward pass is the same: flags drawn beforehand or by the kernel
    # The backward kernels differ by float32 errors, so that single values round to the next bf16 one, 2^-8 of it away. All of
    # them would move a gradient by 2^-8; a hundredth part does, and each of the two layers adds its own.
    for n in a:
        assert float((a[n] - b[n]).norm()) <= 2.0 ** -8 * float(a[n].norm()), n
