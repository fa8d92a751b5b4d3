"""What Gpt2Step hands to the library for a layer: the whole layer in one call where every tensor is what that call takes it
for, single launches otherwise. The library is a stand-in that records its calls, so this runs without a GPU."""
import threading

import pytest
import torch

from conftest import pkg

B, S = 2, 8


class Library:
    """Returns 0 (no scratch needed, no error) from every entry point and remembers the arguments."""

    def __init__(self):
        self.calls = []

    def __getattr__(self, name):
        if not name.startswith("ptj_"):
            raise AttributeError(name)

        def call(*args):
            self.calls.append((name, args))
            return -6 if name == "ptj_gemm_grouped2" else 0  # (a pair of products that does not qualify)

        return call

    def named(self, name):
        return [args for n, args in self.calls if n == name]


@pytest.fixture
def library(monkeypatch):
    ops, lib = pkg("operators"), Library()
    monkeypatch.setattr(ops._lib, "lib", lambda: lib)
    monkeypatch.setattr(ops, "_cuda", lambda t, name="": t.contiguous())
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: False)
    return lib


def engine(dtype=torch.float32):
    g = pkg("gpt2")
    cfg = g.GPT2Config(vocab=64, dim=16, layers=2, heads=2, ffn=32, seq=S)
    step = g.Gpt2Step(cfg, dtype)
    weights = {n: torch.zeros(s, dtype=dtype if g.base_name(n) in g.MATRIX_TENSORS else torch.float32)
               for n, s in cfg.param_shapes()}
    return cfg, step, weights, {n: torch.zeros(s) for n, s in cfg.param_shapes()}


def strided(t):
    """The same shape as columns of a wider matrix."""
    return torch.zeros(*t.shape[:-1], t.shape[-1] + 8, dtype=t.dtype)[..., :t.shape[-1]]


def forward(cfg, step, weights, train=True):
    ids = torch.ones(B, S, dtype=torch.int32)
    seeds = list(range(1 + 3 * cfg.layers))
    logits, acts = step.forward(pkg("gpt2").Weights(cfg, weights), ids, train, seeds)
    return logits, acts, ids, seeds


@pytest.mark.parametrize("other", [None, "strided", "bf16", "smaller"])
def test_a_weight_that_is_not_the_configurations_goes_to_single_launches(library, other):
    cfg, step, weights, _ = engine()
    name = "l1.w2"
    t = weights[name]
    if other is not None:
        weights[name] = {"strided": strided(t), "bf16": t.bfloat16(), "smaller": t[:8].clone()}[other]
    if other == "bf16":
        with pytest.raises(TypeError):  # as a product of two types always did
            forward(cfg, step, weights)
    else:
        forward(cfg, step, weights)
    assert len(library.named("ptj_layer_fwd")) == (cfg.layers if other is None else 0)
    if other == "strided":
        # ptj_gemm(a, b, c, bias, aux, aux_out, M, N, K, lda, ldb, ...)
        (product,) = [a for a in library.named("ptj_gemm") if a[1] == weights[name].data_ptr()]
        assert product[10] == weights[name].stride(0)


@pytest.mark.parametrize("other", [None, "strided", "bf16"])
def test_a_gradient_that_is_not_the_configurations_goes_to_single_launches(library, other):
    cfg, step, weights, grads = engine()
    logits, acts, ids, seeds = forward(cfg, step, weights)
    assert len(library.named("ptj_layer_fwd")) == cfg.layers
    name = "l0.w1"
    if other is not None:
        grads[name] = {"strided": strided(grads[name]), "bf16": grads[name].bfloat16()}[other]
    ready = []
    step.backward(pkg("gpt2").Weights(cfg, weights), grads, logits, acts, ids, True, seeds, ready.extend)
    assert sorted(ready) == sorted(grads)
    assert len(library.named("ptj_layer_bwd_ffn")) == len(library.named("ptj_layer_bwd_attn")) == (
        cfg.layers if other is None else 0)
    if other is not None:
        (product,) = [a for a in library.named("ptj_gemm") if a[2] == grads[name].data_ptr()]
        assert product[11] == grads[name].stride(0) and product[15] == pkg("_lib").PTJ_F32 + (other == "bf16")


def test_threads_in_passes_of_one_shape_keep_their_seeds(library, monkeypatch):
    """The library reads a layer's seeds during the call, while other threads run: here two passes of one engine are both in
    their call before either reads."""
    cfg, step, weights, _ = engine()
    both, seen = threading.Barrier(2, timeout=20), {}

    def layer_fwd(shape, *args):
        both.wait()
        seen.setdefault(threading.current_thread().name, []).append((shape.seed_attn, shape.seed_res1, shape.seed_res2))
        both.wait()
        return 0

    library.ptj_layer_fwd = layer_fwd
    ids = torch.ones(B, S, dtype=torch.int32)
    seeds = {name: [base + i for i in range(1 + 3 * cfg.layers)] for name, base in (("one", 10), ("two", 50))}
    threads = [threading.Thread(target=step.forward, name=name,
                                args=(pkg("gpt2").Weights(cfg, weights), ids, True, seeds[name])) for name in seeds]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert seen == {name: [tuple(s[1 + 3 * l:4 + 3 * l]) for l in range(cfg.layers)] for name, s in seeds.items()}


def test_each_stream_has_a_workspace_of_its_own(library, monkeypatch):
    """... and a recorded graph one that serves nothing else, and that stays when a larger one takes its place."""
    cfg, step, weights, _ = engine()
    now = {"stream": 1, "recording": False, "bytes": 1 << 12}
    monkeypatch.setattr(pkg("operators"), "_stream", lambda: now["stream"])
    monkeypatch.setattr(torch.cuda, "is_current_stream_capturing", lambda: now["recording"])
    library.ptj_layer_workspace_bytes = lambda *a: now["bytes"]

    def workspace(**kw):
        now.update(kw)
        step._plans.clear()
        library.calls.clear()
        forward(cfg, step, weights)
        used = {a[5:7] for a in library.named("ptj_layer_fwd")}
        assert len(used) == 1
        return used.pop()

    first, second, recorded = workspace(), workspace(stream=2), workspace(recording=True)
    assert len({first[0], second[0], recorded[0]}) == 3
    assert workspace(stream=1, recording=False) == first and workspace(stream=2) == second
    larger = workspace(recording=True, bytes=1 << 14)
    assert larger[1] == 1 << 14 and larger[0] != recorded[0]
    assert [t.data_ptr() for t in step._held] == [recorded[0], larger[0]]
    step.release_workspaces()
    assert workspace() == larger and workspace(recording=False)[0] not in (recorded[0], larger[0])


def test_a_pass_that_finds_no_memory_runs_without_what_only_makes_it_faster(library, monkeypatch):
    """Keep flags and the larger workspace are given up, in the forward pass wherever memory ran out, then in the backward
    pass; the gradients' own buffer comes before the workspace."""
    cfg, step, weights, grads = engine(torch.bfloat16)
    big, limit, real = 1 << 30, [None], torch.empty

    def empty(*shape, **kw):
        t = real(*shape, **{**kw, "device": "meta"})
        if limit[0] is not None and t.numel() * t.element_size() >= limit[0]:
            raise torch.OutOfMemoryError("no room")
        return t if t.numel() * t.element_size() >= big else real(*shape, **kw)

    monkeypatch.setattr(torch, "empty", empty)
    library.ptj_layer_keep_bits_bytes = lambda shape: big
    library.ptj_layer_workspace_bytes = lambda shape, backward, products: big if products else 256
    _, acts, _, _ = forward(cfg, step, weights)
    calls = library.named("ptj_layer_fwd")
    assert len(calls) == cfg.layers and all(a[2].keep_bits and a[6] == big for a in calls)
    library.calls.clear()
    limit[0] = big
    logits, acts, ids, seeds = forward(cfg, step, weights)
    calls = library.named("ptj_layer_fwd")
    assert len(calls) == cfg.layers and all(not a[2].keep_bits and a[6] == 256 for a in calls)
    step.backward(pkg("gpt2").Weights(cfg, weights), grads, logits, acts, ids, True, seeds)
    assert [a[-2] for a in library.named("ptj_layer_bwd_attn")] == [256] * cfg.layers


def test_attention_backward_without_room_for_its_workspace(monkeypatch):
    """Shapes that the general kernels can take run there; whole tiles of 64-wide heads say that memory ran out."""
    ops, calls = pkg("operators"), []

    class Library:
        def ptj_attn_bwd_workspace_bytes(self, *a):
            return 1 << 40

        def ptj_attn_bwd(self, *a):
            calls.append(a)
            return 0

    def empty(*a, **kw):
        raise torch.OutOfMemoryError("no room")

    monkeypatch.setattr(ops._lib, "lib", Library)
    monkeypatch.setattr(ops, "_stream", lambda: 0)
    monkeypatch.setattr(ops, "attn_bwd_workspace", empty)
    for N, D, runs in ((100, 64, True), (128, 32, True), (128, 64, False)):
        t = torch.ones(1, 1, N, D, dtype=torch.bfloat16)
        m = torch.ones(1, 1, N)
        calls.clear()
        if not runs:
            with pytest.raises(torch.OutOfMemoryError):
                ops.attn_bwd(t, t, t, t, t, m, m, t, t, t, True, 1)
        else:
            ops.attn_bwd(t, t, t, t, t, m, m, t, t, t, True, 1)
            assert [c[-4:-2] for c in calls] == [(None, 0)]
