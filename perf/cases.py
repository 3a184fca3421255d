"""What the framework is timed on: training steps, generation, scoring and single operators, called
as a user's program calls them.

`listed()` holds the fixed cases and `draw()` makes more of the same ranges. `prepare()` builds what
such a program has in hand before the call (model, optimizer, inputs on the GPU), `run()` makes one
pass, `work()` counts the bytes and operations the pass cannot do without, `tolerance()` says how far
another correct implementation at the same precision may be off.

Kinds of cases:
  train      one optimizer step under the Accelerator: zero_grad, forward, loss, backward, clip, AdamW
  generate   model.generate(): greedy sampling with the key/value cache, fp32 weights, ids on the host
  decode     serving with given tokens: a prompt fills the cache, then one token per step; logits of
             every step
  score      logits of whole sequences without a graph (evaluation)
  attention  scaled-dot-product attention, forward and backward
  linear     a Linear layer with bias and GELU, forward and backward
  rows       the row-wise operators (LayerNorm, RMSNorm, softmax, GELU), forward and backward
"""
import contextlib
import math

import numpy as np
import torch

import mytorch_b200 as mt
from mytorch_b200 import fused_ops as K
from mytorch_b200.array import as_device_array
from mytorch_b200.gpt2 import GPT2, Cache, GPT2Config
from mytorch_b200.nanochat_gpt import GPT, GPTConfig, KVCache

SIZE = {"float32": 4, "float16": 2, "bfloat16": 2}


# ------------------------------------------------------------------- cases ----
def _gpt2(kind, name, dtype, batch, seq, blocks=12, width=768, heads=12, vocab=50304, **more):
    return dict(name=name, kind=kind, model="gpt2", dtype=dtype, batch=batch, seq=seq, blocks=blocks, width=width,
                heads=heads, kv_heads=heads, vocab=vocab, **more)


def _nano(kind, name, dtype, batch, seq, blocks, width=1280, heads=10, kv_heads=10, vocab=65536, **more):
    return dict(name=name, kind=kind, model="nanochat", dtype=dtype, batch=batch, seq=seq, blocks=blocks, width=width,
                heads=heads, kv_heads=kv_heads, vocab=vocab, **more)


def listed():
    return [
        # The first run of every user and of the tests: a character-level model in fp32, many small launches.
        _gpt2("train", "train_tiny_fp32", "float32", 16, 256, blocks=4, width=256, heads=4, vocab=65, loss="mean"),
        # The benchmark's default workload: GPT-2 124M, fp16 mixed precision, padded vocabulary, 16 x 1024 tokens.
        _gpt2("train", "train_gpt2_fp16", "float16", 16, 1024, loss="fused"),
        # The same model as GPT2Config() makes it: the tokenizer's own 50257 entries, a ragged batch, bf16,
        # the plain loss that keeps the logits.
        _gpt2("train", "train_gpt2_bf16_ragged", "bfloat16", 5, 777, vocab=50257, loss="mean"),
        # The d20 model's width and context (10 heads of 128, 65536 entries, rotary, soft-capped loss), four of
        # its blocks: the ordinary large training step.
        _nano("train", "train_nanochat_fp16", "float16", 8, 2048, 4, loss="fused"),
        # A memory-tight run of the same width: grouped-query heads, gradient checkpointing, chunked head, bf16,
        # a sequence that no tile divides.
        _nano("train", "train_nanochat_gqa_bf16", "bfloat16", 2, 1531, 4, kv_heads=2, loss="chunked"),
        # One user at the prompt: greedy generation from the model as its constructor leaves it (fp32).
        _gpt2("generate", "generate_gpt2_fp32", "float32", 1, 19, vocab=50257, new=24),
        # Serving a small batch in half precision, short prompts.
        _gpt2("decode", "decode_gpt2_fp16", "float16", 8, 128, new=16),
        # Serving a full batch with grouped-query heads and rotary positions, longer prompts.
        _nano("decode", "decode_nanochat_gqa_bf16", "bfloat16", 32, 301, 8, kv_heads=2, new=16),
        # Scoring documents: logits of every position, no graph.
        _gpt2("score", "score_gpt2_fp16", "float16", 4, 1000),
        # The operator suite's attention in full precision.
        dict(name="attention_fp32", kind="attention", dtype="float32", batch=8, heads=12, kv_heads=12, seq=1024,
             head_dim=64, causal=True),
        # The operator suite's matrix product as a layer, in full precision.
        dict(name="linear_fp32", kind="linear", dtype="float32", rows=8192, inner=768, outer=3072),
        # The operator suite's row-wise operators.
        dict(name="rows_fp16", kind="rows", dtype="float16", rows=16384, cols=1024),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["train", "train", "train", "generate", "decode", "decode", "score", "attention", "attention",
                       "linear", "linear", "rows"])
    half = rng.choice(["float16", "bfloat16"])
    if kind == "attention":
        dtype = rng.choice(["float32", half, half])
        heads = rng.choice([2, 4, 6, 10, 12])
        c = dict(kind=kind, dtype=dtype, batch=0, heads=heads, kv_heads=rng.choice([heads, heads, 2]),
                 seq=_log(rng, 64, 1024 if dtype == "float32" else 4096), head_dim=rng.choice([32, 64, 64, 96, 128, 128]),
                 causal=rng.random() < 0.75)
        # head sizes that tensor-core tiles do not fit take the full-precision kernels
        cap = 5e10 if dtype != "float32" and c["head_dim"] in (64, 128) else 1.2e10
        per = 7.0 * heads * c["seq"] ** 2 * c["head_dim"]
        c["batch"] = max(1, min(16, int(_log(rng, cap / 20, cap) / per)))
        return c
    if kind == "linear":
        dtype = rng.choice(["float32", half, half])
        c = dict(kind=kind, dtype=dtype, rows=_log(rng, 1, 16384), inner=_log(rng, 64, 4096), outer=_log(rng, 64, 4096))
        if rng.random() < 0.6:      # the widths that models have; the others are odd ones
            c["inner"], c["outer"] = (max(64, c[k] // 64 * 64) for k in ("inner", "outer"))
        c["rows"] = min(c["rows"], max(1, int(6e10 / (c["inner"] * c["outer"]))))
        return c
    if kind == "rows":
        cols = _log(rng, 32, 8192)
        return dict(kind=kind, dtype=rng.choice(["float32", half, half]),
                    rows=min(_log(rng, 16, 65536), int(4e7 / cols)), cols=cols)
    nano = rng.random() < 0.4
    if nano:
        width = rng.choice([640, 1280])
        heads = width // 128
        make = lambda *a, **k: _nano(kind, "", *a, width=width, heads=heads, kv_heads=rng.choice([heads, heads, 1]),
                                     vocab=rng.choice([4096, 32768, 65536]), **k)
    else:
        width = rng.choice([256, 384, 768, 768])
        make = lambda *a, **k: _gpt2(kind, "", *a, width=width, heads=width // 64,
                                     vocab=rng.choice([65, 4096, 50257, 50304]), **k)
    blocks = rng.randint(2, 6)
    seq = _log(rng, 24, 2000 if nano else 1000)
    if kind == "train":
        dtype = rng.choice(["float32", half, half, half])
        tokens = _log(rng, 64, 2000 if dtype == "float32" else 12000)
        c = make(dtype, max(1, tokens // seq), seq, blocks=blocks, loss=rng.choice(["mean", "fused"] + ["chunked"] * nano))
    elif kind == "score":
        c = make(rng.choice(["float32", half]), 1, min(seq, 1000), blocks=blocks)
        c["batch"] = max(1, _log(rng, 32, 600 if c["dtype"] == "float32" else 4000) // c["seq"])
    elif kind == "generate":
        c = make("float32", rng.choice([1, 1, 2, 4]), _log(rng, 4, 200), blocks=blocks, new=rng.randint(8, 24))
    else:
        c = make(half, _log(rng, 1, 32), _log(rng, 8, 500), blocks=blocks, new=rng.randint(6, 16))
    del c["name"]
    return c


# ----------------------------------------------------------------- prepare ----
@contextlib.contextmanager
def _no_host_draws():
    """The model constructors draw every weight on the host, several times over: seconds for a
    model whose step takes milliseconds. `_weights` replaces them from the seed on the GPU, so the
    constructors get zeros meanwhile."""
    names = ("normal", "uniform", "randn")
    saved = {n: getattr(np.random, n) for n in names}
    zeros = lambda shape: np.broadcast_to(np.float32(0), shape)
    np.random.normal = np.random.uniform = lambda a=0.0, b=1.0, size=(): zeros(size)
    np.random.randn = lambda *shape: zeros(shape)
    try:
        yield
    finally:
        for n, f in saved.items():
            setattr(np.random, n, f)


class _Bits:
    """bf16 device memory described to torch as 16-bit integers."""

    def __init__(self, a):
        self.array = a
        self.__cuda_array_interface__ = dict(a.__cuda_array_interface__, typestr="<i2")


def _torch(a):
    """A framework array (or Tensor) as a torch tensor over the same memory."""
    a = getattr(a, "data", a)
    if a.dtype == "bfloat16":
        return torch.as_tensor(_Bits(a), device="cuda").view(torch.bfloat16)
    return torch.as_tensor(a, device="cuda")


def _array(t, dtype=None):
    """A torch tensor's values as a framework array (of `dtype`)."""
    t = t.contiguous()
    torch.cuda.synchronize()
    a = as_device_array(t).copy()
    a = a if dtype is None else a.astype(dtype)
    mt.array.synchronize()
    return a


def _model(case, gen, seq):
    with _no_host_draws():
        if case["model"] == "gpt2":
            model = GPT2(GPT2Config(vocab_size=case["vocab"], max_seq_len=max(seq, 64), embed_dim=case["width"],
                                    num_blocks=case["blocks"], num_heads=case["heads"]))
        else:
            model = GPT(GPTConfig(vocab_size=case["vocab"], max_seq_len=max(seq, 64), embed_dim=case["width"],
                                  num_blocks=case["blocks"], num_q_heads=case["heads"], num_kv_heads=case["kv_heads"]))
    torch.cuda.synchronize()
    _weights(case, model, gen)
    torch.cuda.synchronize()
    return model


def _weights(case, model, gen):
    """Weights of the sizes that training leaves: GPT-2's N(0, 0.02) with smaller output projections
    and larger position rows, 1/sqrt(fan_in) for the nanochat layers, norm weights around one."""
    for name, p in model.named_parameters():
        t = _torch(p)
        if t.dim() < 2:
            t.copy_(1.0 + 0.1 * torch.randn(t.shape, generator=gen, device="cuda"))
            continue
        if case["model"] == "gpt2":
            std = 0.1 if "position" in name else 0.02 / math.sqrt(2 * case["blocks"]) if "out_proj" in name else 0.02
        else:
            std = 0.02 if "embeddings" in name else min(1.0, math.sqrt(t.shape[0] / t.shape[1])) / math.sqrt(t.shape[1])
        t.normal_(0.0, std, generator=gen)


def _ids(case, gen, shape):
    return torch.randint(0, case["vocab"], shape, generator=gen, device="cuda", dtype=torch.int32)


def _tokens(ids):
    return mt.Tensor(_array(ids))


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return {"train": _prepare_train, "generate": _prepare_generate, "decode": _prepare_decode, "score": _prepare_score,
            "attention": _prepare_attention, "linear": _prepare_linear, "rows": _prepare_rows}[case["kind"]](case, gen)


def _prepare_train(case, gen):
    ids = _ids(case, gen, (case["batch"], case["seq"] + 1))
    x, y = _tokens(ids[:, :-1]), _tokens(ids[:, 1:])
    acc = mt.Accelerator(num_gpus=1, rank=0, mixed_precision=case["dtype"] != "float32",
                         half_dtype=case["dtype"] if case["dtype"] != "float32" else "float16")
    model = _model(case, gen, case["seq"])
    decay = [p for _, p in model.named_parameters() if len(p.shape) >= 2]
    rest = [p for _, p in model.named_parameters() if len(p.shape) < 2]
    groups = [{"params": decay, "weight_decay": 0.1}] + ([{"params": rest, "weight_decay": 0.0}] if rest else [])
    opt = mt.optim.AdamW(groups, lr=3e-4, beta1=0.9, beta2=0.95)
    model, opt = acc.prepare(model, opt)
    if case["model"] == "gpt2":
        loss_fn = mt.nn.CrossEntropyLoss(fused_backward=case["loss"] == "fused")
        loss_of = lambda x, y: loss_fn(model(x), y)
    else:
        model.loss_mode = {"mean": "logits"}.get(case["loss"], case["loss"])
        if case["loss"] == "chunked":
            model.enable_gradient_checkpointing()
        loss_of = lambda x, y: model(x, y)[1]
    flat = acc._flat       # the parameters, gradients and moments, each kind in one buffer
    mt.array.synchronize()
    return dict(run=_run_train, acc=acc, opt=opt, loss_of=loss_of, x=x, y=y,
                hint=acc.scaler.scale_dev,
                buffers={k: _torch(getattr(flat, k)) for k in ("master", "grad", "m", "v")})


def _run_train(s):
    acc, opt = s["acc"], s["opt"]
    mt.Tensor.loss_grad_hint = s["hint"]     # the latest Accelerator announces its own; several live here
    opt.zero_grad()
    loss = s["loss_of"](s["x"], s["y"])
    acc.backward(loss)
    acc.clip_grad_norm_(1.0)
    opt.step()
    return dict(s["buffers"], loss=_torch(loss))


def _prepare_generate(case, gen):
    model = _model(case, gen, case["seq"] + case["new"])
    return dict(run=_run_generate, model=model, ids=_ids(case, gen, (case["batch"], case["seq"])).cpu().numpy(), new=case["new"])


def _run_generate(s):
    return s["model"].generate(s["ids"], s["new"], temperature=0)


def _half_model(case, gen, seq):
    model = _model(case, gen, seq)
    for p in model.parameters():
        p.astype(case["dtype"])
    model.eval()
    return model


def _prepare_decode(case, gen):
    total = case["seq"] + case["new"]
    model = _half_model(case, gen, total)
    ids = _ids(case, gen, (case["batch"], total))
    feeds = [_tokens(ids[:, :case["seq"]])] + [_tokens(ids[:, t:t + 1]) for t in range(case["seq"], total)]
    if case["model"] == "gpt2":
        new_cache = lambda: Cache(model.config)
        step = lambda x, cache: model(x, cache=cache)[0]
    else:
        kept = KVCache(case["batch"], case["kv_heads"], total, case["width"] // case["heads"], case["blocks"])

        def new_cache():
            kept.reset()
            return kept
        step = lambda x, cache: model(x, None, cache=cache)[0]
    return dict(run=_run_decode, step=step, new_cache=new_cache, feeds=feeds)


def _run_decode(s):
    cache = s["new_cache"]()
    with mt.no_grad():
        return [_torch(s["step"](x, cache)) for x in s["feeds"]]


def _prepare_score(case, gen):
    model = _half_model(case, gen, case["seq"])
    x = _tokens(_ids(case, gen, (case["batch"], case["seq"])))
    return dict(run=_run_score, model=model, nano=case["model"] == "nanochat", x=x)


def _run_score(s):
    with mt.no_grad():
        out = s["model"](s["x"])
        return _torch(out[0] if s["nano"] else out)


def _prepare_attention(case, gen):
    B, H, Hk, S, D = (case[k] for k in ("batch", "heads", "kv_heads", "seq", "head_dim"))
    make = lambda h: _array(torch.randn((B, h, S, D), generator=gen, device="cuda"), case["dtype"])
    return dict(run=_run_attention, q=make(H), k=make(Hk), v=make(Hk), d_o=make(H), causal=case["causal"])


def _run_attention(s):
    q, k, v, o, lse = K.fused_sdpa_forward(s["q"], s["k"], s["v"], causal=s["causal"])
    dq, dk, dv = K.fused_sdpa_backward(s["d_o"], q, k, v, o, lse, causal=s["causal"])
    return {n: _torch(a) for n, a in (("o", o), ("lse", lse), ("dq", dq), ("dk", dk), ("dv", dv))}


def _prepare_linear(case, gen):
    R, I, O = case["rows"], case["inner"], case["outer"]
    with _no_host_draws():
        layer = mt.nn.Linear(I, O, bias=True, act_func="gelu")
    layer.weight.data = _array(torch.randn((O, I), generator=gen, device="cuda") / math.sqrt(I), case["dtype"])
    layer.bias.data = _array(torch.randn((O,), generator=gen, device="cuda") * 0.1, case["dtype"])
    x = mt.Tensor(_array(torch.randn((R, I), generator=gen, device="cuda"), case["dtype"]), requires_grad=True)
    dy = _array(torch.randn((R, O), generator=gen, device="cuda"), case["dtype"])
    return dict(run=_run_linear, layer=layer, x=x, dy=dy)


def _run_linear(s):
    layer, x = s["layer"], s["x"]
    layer.zero_grad()
    x.grad = None
    y = layer(x)
    y.backward(s["dy"])
    return {"y": _torch(y), "dx": _torch(x.grad), "dw": _torch(layer.weight.grad), "db": _torch(layer.bias.grad)}


def _prepare_rows(case, gen):
    R, C = case["rows"], case["cols"]
    make = lambda *shape: torch.randn(shape, generator=gen, device="cuda")
    return dict(run=_run_rows, x=_array(make(R, C), case["dtype"]), dy=_array(make(R, C), case["dtype"]),
                gamma=_array(1.0 + 0.1 * make(C), case["dtype"]), beta=_array(0.1 * make(C), case["dtype"]))


def _run_rows(s):
    x, dy, gamma, beta = s["x"], s["dy"], s["gamma"], s["beta"]
    out = {}
    y, mean, rstd = K.fused_layernorm_forward(x, gamma, beta)
    out["ln"] = (y, mean, rstd, *K.fused_layernorm_backward(x, mean, rstd, dy, gamma, beta))
    y, rstd = K.fused_rmsnorm_forward(x, gamma)
    out["rms"] = (y, rstd, *K.fused_rmsnorm_backward(x, rstd, dy, gamma))
    p = K.fused_softmax_forward(x)
    out["softmax"] = (p, K.fused_softmax_backward(dy, p))
    out["gelu"] = (K.fused_activation_forward(x, "gelu"), K.fused_activation_backward(x, dy, "gelu"))
    return {k: [_torch(a) for a in v] for k, v in out.items()}


def run(state):
    return state["run"](state)


# -------------------------------------------------------------------- work ----
def _counts(case):
    """(weights outside the embedding tables and the head, weights of the head, all weights)."""
    d, L = case["width"], case["blocks"]
    kv = d * case["kv_heads"] // case["heads"]
    body = L * (2 * d * d + 2 * d * kv + 8 * d * d)
    head = d * case["vocab"]
    gpt2 = case["model"] == "gpt2"
    return body, head, body + head * (1 if gpt2 else 2) + (case["seq"] * d if gpt2 else 0)


def work(case):
    kind, e = case["kind"], SIZE[case["dtype"]]
    if kind == "attention":
        q = case["batch"] * case["heads"] * case["seq"] * case["head_dim"]
        kv = q * case["kv_heads"] // case["heads"]
        mac = q * case["seq"] * (0.5 if case["causal"] else 1.0)
        # q, k, v, dO in; o, dq, dk, dv out; two products forward, five backward
        return {"bytes": float(e * (4 * q + 4 * kv)), "flops": 14.0 * mac}
    if kind == "linear":
        R, I, O = case["rows"], case["inner"], case["outer"]
        # x, w, dy in; y, dx out; dw in fp32 out
        return {"bytes": float(e * (2 * R * I + 2 * R * O + I * O) + 4 * I * O), "flops": 6.0 * R * I * O}
    if kind == "rows":
        n = case["rows"] * case["cols"]
        # each operator: forward reads one tensor and writes one, backward reads two and writes one
        return {"bytes": float(4 * 5 * n * e), "flops": 60.0 * n}
    body, head, every = _counts(case)
    B, T, d, L = case["batch"], case["seq"], case["width"], case["blocks"]
    attn = lambda tokens, keys: 4.0 * L * d * tokens * keys
    kv_row = 2 * L * d * case["kv_heads"] // case["heads"] * e
    if kind == "train":
        tok = B * T
        # AdamW: weight, gradient and two moments read, weight and moments written, half copy written and read
        return {"bytes": float(every * (28 + (4 if e == 2 else 0))), "flops": 6.0 * tok * (body + head) + 3 * attn(tok, T / 2)}
    if kind == "score":
        return {"bytes": float(every * e + B * T * case["vocab"] * e), "flops": 2.0 * B * T * (body + head) + attn(B * T, T / 2)}
    n = case["new"]
    steps = n if kind == "decode" else n - 1              # generate's first token comes out of the prompt pass
    heads_needed = B * (T + n) if kind == "decode" else B * n
    moved = (1 + steps) * (body + head) * e + B * kv_row * steps * (T + steps / 2)
    if kind == "decode":
        moved += heads_needed * case["vocab"] * e
    return {"bytes": float(moved), "flops": 2.0 * (B * (T + steps) * body + heads_needed * head)
            + attn(B * T, T / 2) + attn(B * steps, T + steps / 2)}


def tolerance(case):
    kind, dtype = case["kind"], case["dtype"]
    if kind == "generate":
        return {"rel": 0.0, "differ": 0.01}                # token ids: only a tie of the two best logits may differ
    if kind == "train":
        # Rounding of every layer's activations, twice in the squared moment. An AdamW step has a
        # size of lr whatever the gradient's: where a gradient is all rounding, the weight moves by
        # up to 2 lr = 6e-4 either way, 0.03 of N(0, 0.02) weights.
        return {"float32": {"rel": 1e-4, "max": 0.05}, "float16": {"rel": 1e-2}, "bfloat16": {"rel": 2e-2}}[dtype]
    if kind in ("decode", "score"):
        return {"rel": {"float32": 2e-5, "float16": 5e-3, "bfloat16": 1e-2}[dtype]}
    return {"rel": {"float32": 1e-5, "float16": 2e-3, "bfloat16": 1e-2}[dtype]}
