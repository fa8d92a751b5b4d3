"""What Gpt2Step hands to the library for a layer: the whole layer in one call where every tensor is what that call takes it
for, single launches otherwise. The library is a stand-in that records its calls, so this runs without a GPU."""
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
    step._ws = torch.zeros(1 << 16)
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
