"""Timed work of the GPT-2 training framework, as a user's program has it done, through the public entry points.

Each case is a dict of plain values with a ``kind``:

* ``train``      one ``Trainer.step`` from pinned host token ids: forward, backward, clip, AdamW (bf16 compute)
* ``micro_step`` the reference-shaped pytree path: ``t_loss_bkwd3_t`` and, for float32 parameters, ``adam_w_in_place``
* ``forward``    evaluation forward over whole sequences (prefill), ``t_gpt2_forward(train=False)``
* ``score``      ``log_probs``: per-sequence log-probabilities of given continuations
* ``predict``    greedy decoding, ``predict``
* ``attention``  the attention operator, forward and backward, on ``qkv[B, H, 3, N, D]``
* ``loss``       the cross-entropy operator, forward and backward, on contiguous logits
* ``layernorm``  the LayerNorm operator, forward and both backward launchers

Inputs are synthetic: Zipf(1.1) token ids (0 is the padding id), seeded random weights of the architecture.
"""
import importlib
import math

import torch

ptj = importlib.import_module("pre-tjax_b200")
ops, gpt2, trainer, evaluate, optimizer = ptj.operators, ptj.gpt2, ptj.trainer, ptj.evaluate, ptj.optimizer

DTYPES = {"bf16": torch.bfloat16, "f32": torch.float32}
MODEL = ("vocab", "dim", "layers", "heads", "ffn", "seq")
SMALL = dict(dim=768, layers=12, heads=12, ffn=3072)


def listed():
    medium = dict(dim=1024, layers=24, heads=16, ffn=4096)
    return [
        # the toy model a developer steps through: 128 tokens per row, latency and launches are all there is
        dict(name="train tiny", kind="train", vocab=1024, dim=128, layers=2, heads=4, ffn=512, seq=128, batch=4,
             dropout=0.0, graph=False, packed=False),
        # the headline: GPT-2 small pre-training at 8 x 1024 tokens per GPU, step replayed from a graph
        dict(name="train small", kind="train", vocab=50257, seq=1024, batch=8, dropout=0.1, graph=True, packed=False,
             **SMALL),
        # the same model fed by the collator that packs documents into rows (document masks, padded tails)
        dict(name="train small packed", kind="train", vocab=50257, seq=1024, batch=8, dropout=0.1, graph=True,
             packed=True, **SMALL),
        # the largest configuration: GPT-2 medium at 16 x 1024 tokens per GPU
        dict(name="train medium", kind="train", vocab=50257, seq=1024, batch=16, dropout=0.1, graph=True, packed=False,
             **medium),
        # drop-in use of the reference's float32 pytree functions at its own vocabulary, row length and micro-batch
        dict(name="micro step f32", kind="micro_step", dtype="f32", vocab=35374, dim=768, layers=4, heads=12, ffn=3072,
             seq=512, batch=8, packed=True),
        # prefill: logits of three full-length sequences with bf16 weights
        dict(name="forward small", kind="forward", dtype="bf16", vocab=50257, seq=1024, batch=3, **SMALL),
        # multiple-choice scoring between training steps, on the float32 master weights: four endings of a context
        dict(name="score small f32", kind="score", dtype="f32", vocab=35374, seq=512, batch=4, **SMALL),
        # samples drawn during training to look at, on the float32 master weights
        dict(name="predict small f32", kind="predict", dtype="f32", vocab=35374, seq=128, batch=2, **SMALL),
        # the attention microbenchmark shape, with dropout
        dict(name="attention 1024", kind="attention", dtype="bf16", batch=8, heads=12, seq=1024, d_head=64, packed=False),
        # a row length that is not a multiple of any tile
        dict(name="attention ragged", kind="attention", dtype="bf16", batch=4, heads=12, seq=500, d_head=64, packed=False),
        # loss of a full micro-batch over the whole vocabulary, rows without padding between them
        dict(name="loss 50257", kind="loss", dtype="bf16", rows=8192, vocab=50257),
        # a single normalisation, forward and backward, at the reference's own benchmark shape
        dict(name="layernorm", kind="layernorm", dtype="bf16", rows=4096, dim=768),
    ]


# ---- drawn cases ------------------------------------------------------------------------------------------------------
MOST_TRAIN = 6.0e12   # parameters x tokens of a drawn training step (the largest listed one: 5.8e12)
MOST_F32 = 2.5e11     # ... of a float32 micro-step or scoring pass
MOST_PREDICT = 6.0e12  # parameters x batch x seq^2 of a drawn decoding


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _seq(rng, hi):
    n = _log_int(rng, 64, hi)
    return max(64, n // 128 * 128) if rng.random() < 0.5 else n


def _model(rng, most_layers, most_seq):
    d_head = rng.choice([32, 64, 64, 64, 128])
    heads = max(1, _log_int(rng, 128, 1024) // d_head)
    dim = heads * d_head
    ffn = 4 * dim if rng.random() < 0.7 else int(dim * rng.uniform(2.0, 4.0)) // 8 * 8
    return dict(vocab=_log_int(rng, 1000, 50257), dim=dim, layers=_log_int(rng, 1, most_layers), heads=heads, ffn=ffn,
                seq=_seq(rng, most_seq))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "micro_step", "micro_step", "forward", "score", "predict",
                       "attention", "attention", "loss", "layernorm"])
    while True:
        if kind == "train":
            c = dict(kind=kind, **_model(rng, 24, 1024), batch=_log_int(rng, 1, 16),
                     dropout=rng.choice([0.0, 0.1, 0.1]), graph=rng.random() < 0.5, packed=rng.random() < 0.3)
            cost, most = _params(c) * c["batch"] * c["seq"], MOST_TRAIN
        elif kind == "micro_step":
            c = dict(kind=kind, dtype=rng.choice(["f32", "f32", "bf16"]), **_model(rng, 4, 1024),
                     batch=_log_int(rng, 1, 8), packed=rng.random() < 0.7)
            cost, most = _params(c) * c["batch"] * c["seq"], MOST_F32
        elif kind == "forward":
            c = dict(kind=kind, dtype="bf16", **_model(rng, 12, 1024), batch=_log_int(rng, 1, 8))
            cost, most = _params(c) * c["batch"] * c["seq"], MOST_TRAIN
        elif kind == "score":
            c = dict(kind=kind, dtype=rng.choice(["f32", "bf16"]), **_model(rng, 12, 512), batch=_log_int(rng, 1, 8))
            cost, most = _params(c) * c["batch"] * c["seq"], MOST_F32
        elif kind == "predict":
            c = dict(kind=kind, dtype="f32", **_model(rng, 12, 256), batch=_log_int(rng, 1, 4))
            cost, most = _params(c) * c["batch"] * c["seq"] ** 2, MOST_PREDICT
        elif kind == "attention":
            c = dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "f32"]), batch=_log_int(rng, 1, 8),
                     heads=_log_int(rng, 1, 16), seq=_seq(rng, 1024), d_head=rng.choice([32, 64, 64, 128]),
                     packed=rng.random() < 0.3)
            cost, most = 1, 1
        elif kind == "loss":
            c = dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "f32"]), rows=_log_int(rng, 256, 8192),
                     vocab=_log_int(rng, 1000, 50257))
            cost, most = 1, 1
        else:
            c = dict(kind=kind, dtype=rng.choice(["bf16", "bf16", "f32"]), rows=_log_int(rng, 128, 16384),
                     dim=8 * _log_int(rng, 16, 256))
            cost, most = 1, 1
        if cost <= most:
            return c


# ---- inputs -----------------------------------------------------------------------------------------------------------
def _config(case):
    return gpt2.GPT2Config(**{k: case[k] for k in MODEL}, dropout=case.get("dropout", ops.DROPOUT_RATE))


def _params(case):
    return _config(case).num_params()


def _weights(cfg, gen, dtype, residual=None):
    """Parameter pytree on the GPU: N(0, 0.02) matrices, residual projections scaled by 1/sqrt(2 L) (or of the given
    deviation), small non-zero vectors; vectors stay float32."""
    res = optimizer.INIT_SCALE / math.sqrt(2 * cfg.layers) if residual is None else residual
    flat = []
    for name, shape in cfg.param_shapes():
        base = gpt2.base_name(name)
        t = torch.randn(shape, generator=gen, device="cuda")
        if base in gpt2.MATRIX_TENSORS:
            t = (t.mul_(res if base in ("w_o", "w2") else optimizer.INIT_SCALE)).to(dtype)
        else:
            t = t.mul_(0.02).add_(1.0 if base[0] == "g" else 0.0)
        flat.append(t)
    return gpt2.unflatten_like(flat, cfg)


def _ids(vocab, shape, gen):
    """int32 token ids with P(id = r) proportional to r^-1.1, r = 1..vocab-1."""
    cdf = torch.cumsum(torch.arange(1, vocab, device="cuda", dtype=torch.float64).pow(-1.1), 0)
    u = torch.rand(shape, generator=gen, device="cuda", dtype=torch.float64) * cdf[-1]
    return (torch.searchsorted(cdf, u).clamp_(max=vocab - 2) + 1).to(torch.int32)


def _documents(batch, seq, seed):
    """Lengths of the documents packed into each row: about three to a row of 1024 tokens, with a short padded tail."""
    g = torch.Generator().manual_seed(seed)
    rows = []
    for _ in range(batch):
        tail = int(torch.randint(0, max(1, seq // 32), (1,), generator=g))
        left, lens = seq - tail, []
        while left > 0:
            n = int(-350.0 * math.log(1.0 - float(torch.rand(1, generator=g)))) + 16
            lens.append(min(n, left))
            left -= lens[-1]
        rows.append(lens)
    return rows


def _pad_tails(y, lens):
    for b, ls in enumerate(lens):
        y[b, sum(ls) + 1:] = 0
    return y


def _dense_mask(kstart):
    """The collator's boolean [B, N, N] mask of packed rows (True = attend)."""
    n = kstart.shape[1]
    i = torch.arange(n, device=kstart.device)
    return (i.view(1, 1, n) >= kstart.unsqueeze(2)) & (i.view(1, 1, n) <= i.view(1, n, 1))


def _flat_views(cfg, sources):
    """The pytree as views of one flat buffer per kind of state (parameters, first and second moments)."""
    layout = trainer.FlatLayout.build(cfg)
    names = [n for n, _ in cfg.param_shapes()]
    out = []
    for src in sources:
        flat = torch.zeros(layout.total, device="cuda")
        if src is not None:
            for n, t in zip(names, gpt2.flatten_pytree(src)):
                layout.view(flat, n).copy_(t)
        out.append((flat, gpt2.unflatten_like([layout.view(flat, n) for n in names], cfg)))
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    st = dict(kind=kind)
    if kind in ("train", "micro_step", "forward", "score", "predict"):
        cfg = _config(case)
        dtype = DTYPES[case.get("dtype", "f32")]
        # decoding: residual branches that outweigh the token embedding, as in a trained network (at the scale of a
        # fresh one the tied embedding only repeats its input)
        params = _weights(cfg, gen, dtype, residual=8.0 / math.sqrt(cfg.dim) if kind == "predict" else None)
        y = _ids(cfg.vocab, (case["batch"], cfg.seq + 1), gen)
        kstart = None
        if case.get("packed"):
            lens = _documents(case["batch"], cfg.seq, seed)
            kstart = ops.row_kstart_from_lengths(lens, cfg.seq)
            y = _pad_tails(y, lens)
    if kind == "train":
        tc = trainer.TrainConfig.benchmark_recipe(seed=seed % 1000, cuda_graph=case["graph"])
        st.update(trainer=trainer.Trainer(cfg, tc, params=params), y=y.cpu().pin_memory(), kstart=kstart)
    elif kind == "micro_step":
        st.update(params=params, y=y, mask=_dense_mask(kstart) if kstart is not None else None,
                  seeds=trainer.step_seeds(seed % 1000, 0, 0, 1 + 3 * cfg.layers))
        if case["dtype"] == "f32":
            (p, params), (m, mm), (v, vv) = _flat_views(cfg, (params, None, None))
            st.update(params=params, moments=[mm, vv], state=(p, m, v), decay=optimizer.weight_decay_mask(
                [[t if gpt2.is_decayed(n) else torch.zeros_like(t) for n, t in zip(ns, ts)]
                 for ns, ts in zip(gpt2.unflatten_like([n for n, _ in cfg.param_shapes()], cfg), params)]))
    elif kind == "forward":
        st.update(params=params, y=y[:, :-1].contiguous())
    elif kind == "score":
        y[:, -(cfg.seq // 8):] = 0  # endings shorter than the row
        st.update(params=params, y=y)
    elif kind == "predict":
        st.update(params=params, batch=case["batch"], seq=cfg.seq, start=cfg.vocab - 2, end=cfg.vocab - 1)
    elif kind == "attention":
        shape = (case["batch"], case["heads"], 3, case["seq"], case["d_head"])
        qkv = torch.randn(shape, generator=gen, device="cuda").to(DTYPES[case["dtype"]])
        d_o = torch.randn(shape[:2] + shape[3:], generator=gen, device="cuda").to(DTYPES[case["dtype"]])
        mask = None
        if case["packed"]:
            lens = [[*ls[:-1], ls[-1] + case["seq"] - sum(ls)] for ls in _documents(case["batch"], case["seq"], seed)]
            mask = _dense_mask(ops.row_kstart_from_lengths(lens, case["seq"]))
        st.update(qkv=qkv, d_o=d_o, mask=mask, seed=seed)
    elif kind == "loss":
        logits = 2.0 * torch.randn(case["rows"], case["vocab"], generator=gen, device="cuda")
        st.update(logits=logits.to(DTYPES[case["dtype"]]), labels=_ids(case["vocab"], (case["rows"],), gen))
    else:
        x, dy = (torch.randn(case["rows"], case["dim"], generator=gen, device="cuda").to(DTYPES[case["dtype"]])
                 for _ in range(2))
        gamma = 1.0 + 0.1 * torch.randn(case["dim"], generator=gen, device="cuda")
        beta = 0.1 * torch.randn(case["dim"], generator=gen, device="cuda")
        st.update(x=x, dy=dy, layer=(gamma, beta))
    return st


# ---- one pass ---------------------------------------------------------------------------------------------------------
def run(st):
    kind = st["kind"]
    if kind == "train":
        t = st["trainer"]
        stats = t.step(st["y"], row_kstart=st["kstart"])
        return {"stats": stats, "weights": t.p, "gradients": t.g, "moments": (t.m, t.v)}
    if kind == "micro_step":
        grads, stats = gpt2.t_loss_bkwd3_t(st["params"], st["y"], st["mask"], None, True, st["seeds"])
        if "moments" not in st:
            return {"stats": stats, "gradients": grads}
        optimizer.adam_w_in_place(st["params"], grads, 2.5e-4, (0.9, 0.98), 1e-8, st["moments"], 0, 0.01, st["decay"])
        return {"stats": stats, "gradients": grads, "state": st["state"]}
    if kind == "forward":
        return evaluate.t_gpt2_forward(st["params"], st["y"], None, None, False)
    if kind == "score":
        return evaluate.log_probs(st["params"], st["y"])
    if kind == "predict":
        return evaluate.predict(st["params"], st["batch"], None, st["seq"], st["start"], st["end"])
    if kind == "attention":
        out, acts = ops.t_scaled_dot_prod_attn_fwd3_t(st["qkv"], st["mask"], True, st["seed"])
        return out, acts[:2], ops.t_scaled_dot_prod_attn_bkwd3_t(st["d_o"], acts, st["qkv"], st["mask"], True, st["seed"])
    if kind == "loss":
        return ops.t_avg_cross_entropy_loss_bkwd3_t(st["labels"], st["logits"])
    y = ops.t_layernorm_fwd_t(st["layer"], st["x"])
    dx = ops.t_layernorm_bkwd2_x_t(st["dy"], st["layer"], st["x"])
    return y, dx, ops.t_layernorm_bkwd2_p_t(st["dy"], st["layer"], st["x"])


# ---- what a pass cannot do without --------------------------------------------------------------------------------------
def _forward_flops(c):
    """Matrix products and causal attention of one forward pass."""
    tokens = c["batch"] * c["seq"]
    mats = c["layers"] * (4 * c["dim"] ** 2 + 2 * c["dim"] * c["ffn"]) + c["vocab"] * c["dim"]
    return 2.0 * tokens * mats + c["layers"] * 2.0 * c["batch"] * c["dim"] * c["seq"] ** 2


def work(case):
    kind = case["kind"]
    size = 4 if case.get("dtype", "bf16") == "f32" else 2
    if kind == "train":  # float32 weights, gradients and two moments, the bf16 copy that the products read; token ids
        return {"bytes": 30.0 * _params(case) + 4.0 * case["batch"] * (case["seq"] + 1), "flops": 3 * _forward_flops(case)}
    if kind == "micro_step":
        per = 28.0 if size == 4 else 2.0 + 4.0
        return {"bytes": per * _params(case) + 4.0 * case["batch"] * (case["seq"] + 1), "flops": 3 * _forward_flops(case)}
    if kind == "forward":
        return {"bytes": size * (_params(case) + case["batch"] * case["seq"] * case["vocab"]), "flops": _forward_flops(case)}
    if kind == "score":
        return {"bytes": float(size * _params(case)), "flops": _forward_flops(case)}
    if kind == "predict":  # every token waits for the one before it, so each reads the weights again
        body = _params(case) - case["seq"] * case["dim"]
        return {"bytes": 4.0 * body * (case["seq"] - 1), "flops": 2.0 * body * case["batch"] * (case["seq"] - 1)}
    if kind == "attention":
        rows = case["batch"] * case["heads"] * case["seq"]
        return {"bytes": 8.0 * size * rows * case["d_head"] + 8.0 * rows, "flops": 7.0 * rows * case["seq"] * case["d_head"]}
    if kind == "loss":
        return {"bytes": 2.0 * size * case["rows"] * case["vocab"], "flops": 4.0 * case["rows"] * case["vocab"]}
    return {"bytes": 4.0 * size * case["rows"] * case["dim"], "flops": 20.0 * case["rows"] * case["dim"]}


def tolerance(case):
    """About four times the error against float64 (operators, scores) or the measured difference to the same path with
    its sums in another order, worst tensor of the pass."""
    f32 = case.get("dtype", "bf16") == "f32"
    kind = case["kind"]
    if kind == "predict":
        return "exact"  # the arg-max gap of a step is some hundred times the float32 error of its logits
    if kind == "micro_step":
        # float32: 4e-6 for the matrices but 7e-5 for the last LayerNorm's shift, a sum that cancels to a thousandth
        # of its terms; Adam's first step is lr * sign(g), so a weight whose gradient is near zero moves by 7e-3 rms
        return {"rel": 3e-4, "max": 3e-2} if f32 else {"rel": 3e-2}
    if kind == "train":
        return {"rel": 1e-2, "max": 0.3}   # 6e-4 (maximum 6e-2) from the order of sums alone, 3e-3 against float64
    if kind == "forward":
        return {"rel": 2e-2, "max": 0.2}   # 9e-3 against float64
    if kind == "attention":
        return {"rel": 1e-5, "max": 1e-4} if f32 else {"rel": 1.2e-2, "max": 0.35}  # 8e-7 / 3e-3 against float64
    if kind == "score":
        return {"rel": 1e-6} if f32 else {"rel": 3e-4}   # 5e-8 / 6e-5
    if kind == "loss":
        return {"rel": 1e-6, "max": 1e-5} if f32 else {"rel": 5e-4, "max": 2e-2}  # 2e-8 / 1.2e-4
    return {"rel": 1e-6, "max": 1e-5} if f32 else {"rel": 7e-3, "max": 2e-2}  # 1.5e-7 / 1.7e-3
