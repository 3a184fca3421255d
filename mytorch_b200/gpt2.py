"""GPT-2 as wired in the reference (gpt2_trainer/gpt2.py:88-390): learned token
and position embeddings, pre-LayerNorm blocks (attention + GELU MLP, 4x), final
LayerNorm, lm_head tied to the token embedding. Same config fields, module
names and state_dict keys, so checkpoints move between the two.

The attention module reads the
per-head interleaved [q|k|v] projection in place (see F.qkv_attention) and the
embedding pair is one kernel; everything else is the same sequence of ops.
"""
import ctypes as C
from dataclasses import dataclass

import numpy as np

from . import _lib, infer, nn
from .array import DeviceArray, stream
from .nn import functional as F
from .tensor import Tensor


@dataclass
class GPT2Config:          # gpt2_trainer/gpt2.py:12-27
    vocab_size: int = 50257
    max_seq_len: int = 1024
    embed_dim: int = 768
    mlp_ratio: int = 4
    num_blocks: int = 12
    num_heads: int = 12
    mlp_dropout_p: float = 0.0
    attn_dropout_p: float = 0.0
    use_bias: bool = False
    use_layernorm_weight: bool = True
    use_full_auto: bool = False
    use_fused_ops: bool = True


class Cache:
    """Key/value cache of the inference step (gpt2_trainer/gpt2.py:29-86): per layer one
    preallocated ring [B, H, max_seq_len, D] for keys and one for values. `update` appends the new
    rows in place; when the ring is full the oldest row is overwritten, which is the reference's
    drop-the-oldest policy without its concatenate and slice copies (attention does not depend on
    the order in which the cached keys are stored)."""

    def __init__(self, config):
        self.max_seq_len = config.max_seq_len
        self.key_cache = [None] * config.num_blocks
        self.value_cache = [None] * config.num_blocks
        self._appended = [0] * config.num_blocks

    def __repr__(self):
        return f"DynamicCache(Num_Layers: {len(self.key_cache)} | Cached Tokens: {self.get_seq_len()})"

    def get_seq_len(self, layer_idx=0):
        return min(self._appended[layer_idx], self.max_seq_len)

    def reserve(self, blocks, batch, heads, head_dim, dtype):
        """All layers' rings, allocated together when none of them exists yet. False when the cache has
        another number of layers, or its layers do not hold the same number of rows of this shape."""
        n = len(self.key_cache)
        if n != blocks or any(a != self._appended[0] for a in self._appended):
            return False
        shape = (batch, heads, self.max_seq_len, head_dim)
        if all(k is None for k in self.key_cache):
            rings = DeviceArray.empty((2 * n,) + shape, dtype)
            ring = lambda i: rings.rows(i, i + 1).reshape(shape)
            self.key_cache = [ring(2 * i) for i in range(n)]
            self.value_cache = [ring(2 * i + 1) for i in range(n)]
        return all(r is not None and r.shape == shape and r.dtype == dtype for r in self.key_cache + self.value_cache)

    def update(self, k_ptr, v_ptr, strides, batch, heads, n_new, head_dim, dtype, layer_idx):
        """Appends n_new rows read through (ptr, strides) and returns (keys, values, rows held)."""
        if self.key_cache[layer_idx] is None:
            shape = (batch, heads, self.max_seq_len, head_dim)
            self.key_cache[layer_idx] = DeviceArray.empty(shape, dtype)
            self.value_cache[layer_idx] = DeviceArray.empty(shape, dtype)
        kc, vc = self.key_cache[layer_idx], self.value_cache[layer_idx]
        assert kc.shape[0] == batch and kc.dtype == dtype, "cache was created for another batch size or dtype"
        sc = _lib.Strides3(heads * self.max_seq_len * head_dim, self.max_seq_len * head_dim, head_dim)
        _lib.kv_append(k_ptr, v_ptr, kc.ptr, vc.ptr, strides, strides, sc, batch, heads, n_new,
                       self._appended[layer_idx] % self.max_seq_len, self.max_seq_len, head_dim, kc.code, stream())
        self._appended[layer_idx] += n_new
        return kc, vc, self.get_seq_len(layer_idx)


class Embeddings(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.config = config
        self.char_embeddings = nn.Embedding(config.vocab_size, config.embed_dim)
        self.position_embeddings = nn.Embedding(config.max_seq_len, config.embed_dim)

    def forward(self, input_ids, past_length=0):
        if past_length == 0:
            return F.token_position_embedding(input_ids, self.char_embeddings.weight, self.position_embeddings.weight)
        # decoding: positions continue after the cached tokens (gpt2.py:115-117); inference only
        B, T = input_ids.shape
        E = self.config.embed_dim
        assert past_length + T <= self.config.max_seq_len, "position table exhausted"
        x = F.embedding(input_ids, self.char_embeddings.weight).data
        pos = self.position_embeddings.weight.data.rows(past_length, past_length + T)
        _lib.add_rowvec(x.ptr, pos.ptr, x.ptr, B, T * E, x.code, stream())
        return Tensor(x)


class Attention(nn.Module):
    def __init__(self, config):
        super().__init__()
        assert config.embed_dim % config.num_heads == 0
        self.embed_dim, self.num_heads = config.embed_dim, config.num_heads
        self.head_dim = config.embed_dim // config.num_heads
        self.qkv_proj = nn.Linear(self.embed_dim, 3 * self.embed_dim, bias=config.use_bias)
        self.out_proj = nn.Linear(self.embed_dim, self.embed_dim, bias=config.use_bias)
        self.proj_drop = nn.Dropout(config.attn_dropout_p)

    def forward(self, x, residual=None, cache=None, layer_idx=None):
        qkv = self.qkv_proj(x)                                   # [B, T, 3E], per-head [q|k|v]
        if cache is not None and layer_idx is not None:
            out = self._cached_attention(qkv, cache, layer_idx)
        else:
            out = F.qkv_attention(qkv, self.num_heads, is_causal=True)  # [B, T, E]
        # the block's skip connection is added in the projection's GEMM epilogue
        out = F.linear(out, self.out_proj.weight, self.out_proj.bias, residual=residual)
        return self.proj_drop(out)


    def _cached_attention(self, qkv, cache, layer_idx):
        """gpt2.py:179-215: the new keys/values join the cache; an empty cache means this call is
        the prompt (causal attention among its tokens), otherwise the new queries see every cached
        key. Inference only (no graph is recorded)."""
        B, T, _ = qkv.shape
        H, D, E = self.num_heads, self.head_dim, self.embed_dim
        arr = qkv.data
        sin = _lib.Strides3(T * 3 * E, 3 * D, 3 * E)               # q/k/v of head h start at h*3D (+0, +D, +2D)
        past = cache.get_seq_len(layer_idx)
        kc, vc, kv_len = cache.update(arr.ptr + D * arr.itemsize, arr.ptr + 2 * D * arr.itemsize, sin, B, H, T, D,
                                      arr.dtype, layer_idx)
        if past == 0:
            return F.qkv_attention(qkv.detach(), H, is_causal=True)
        out = DeviceArray.empty((B, T, E), arr.dtype)
        sc = _lib.Strides3(H * cache.max_seq_len * D, cache.max_seq_len * D, D)
        _lib.attn_decode(arr.ptr, kc.ptr, vc.ptr, out.ptr, sin, sc, _lib.Strides3(T * E, D, E), B, H, T, kv_len, D,
                         float(D) ** -0.5, -1, arr.code, stream())
        return Tensor(out)


class FeedForward(nn.Module):
    def __init__(self, config):
        super().__init__()
        hidden = config.embed_dim * config.mlp_ratio
        self.intermediate_dense = nn.Linear(config.embed_dim, hidden, bias=config.use_bias, act_func="gelu")
        self.intermediate_dropout = nn.Dropout(config.mlp_dropout_p)
        self.out_proj = nn.Linear(hidden, config.embed_dim, bias=config.use_bias)
        self.output_dropout = nn.Dropout(config.mlp_dropout_p)

    def forward(self, x, residual=None):
        if self.intermediate_dense.bias is None and self.out_proj.bias is None:
            # bias-free (the GPT-2 configuration): one fused node, activation and its
            # derivative live in GEMM epilogues, skip connection added in the last one
            return F.mlp(x, self.intermediate_dense.weight, self.out_proj.weight, "gelu", residual=residual)
        h = self.intermediate_dropout(self.intermediate_dense(x))
        return self.output_dropout(F.linear(h, self.out_proj.weight, self.out_proj.bias, residual=residual))


class TransformerBlock(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.attention = Attention(config)
        self.layernorm1 = nn.LayerNorm(config.embed_dim, weight=config.use_layernorm_weight, bias=config.use_bias)
        self.feedforward = FeedForward(config)
        self.layernorm2 = nn.LayerNorm(config.embed_dim, weight=config.use_layernorm_weight, bias=config.use_bias)

    def forward(self, x, cache=None, layer_idx=None):
        # The skip connections are added in the epilogue of each sublayer's last GEMM.
        x = self.attention(self.layernorm1(x), residual=x, cache=cache, layer_idx=layer_idx)
        x = self.feedforward(self.layernorm2(x), residual=x)
        return x


def _init_weights(module):     # gpt2_trainer/gpt2.py:376-389
    if isinstance(module, nn.Linear):
        nn.init.normal_(module.weight, mean=0.0, std=0.02)
        if module.bias is not None:
            nn.init.zeros_(module.bias)
    elif isinstance(module, nn.Embedding):
        nn.init.normal_(module.weight, mean=0.0, std=0.02)
    elif isinstance(module, nn.LayerNorm):
        if module.weight is not None:
            nn.init.ones_(module.weight)
        if module.bias is not None:
            nn.init.zeros_(module.bias)


def _plan(model):
    """What the library's whole-model forward needs to know of the model as it is now (see
    infer.plan_of); None when it does not cover it."""
    cfg, plain = model.config, infer.plain
    e, lnf, head = model.embeddings, model.final_layer_norm, model.lm_head
    if not (infer.unpatched(_METHODS) and plain(model, GPT2) and plain(e, Embeddings) and plain(lnf, nn.LayerNorm)
            and plain(head, nn.Linear) and head.act_func is None):
        return None
    H, E = cfg.num_heads, cfg.embed_dim
    eps = {lnf.eps}
    found = [e.char_embeddings.weight, e.position_embeddings.weight, lnf.weight, lnf.bias, head.weight, head.bias, None, None]
    for b in model.blocks:
        if not plain(b, TransformerBlock):
            return None
        a, f, n1, n2 = b.attention, b.feedforward, b.layernorm1, b.layernorm2
        if not (plain(a, Attention) and "_cached_attention" not in a.__dict__ and plain(f, FeedForward) and plain(n1, nn.LayerNorm)
                and plain(n2, nn.LayerNorm) and a.num_heads == H and a.embed_dim == E and a.head_dim * H == E):
            return None
        qkv, out, up, down = a.qkv_proj, a.out_proj, f.intermediate_dense, f.out_proj
        if not (plain(qkv, nn.Linear) and plain(out, nn.Linear) and plain(up, nn.Linear) and plain(down, nn.Linear)
                and qkv.act_func is None and out.act_func is None and up.act_func == "gelu" and down.act_func is None):
            return None
        for drop in (a.proj_drop, f.intermediate_dropout, f.output_dropout):
            if not (plain(drop, nn.Dropout) and drop.p == 0.0):
                return None
        eps.update((n1.eps, n2.eps))
        found += [n1.weight, n1.bias, n2.weight, n2.bias, qkv.weight, None, None, out.weight, up.weight, down.weight,
                  qkv.bias, None, None, out.bias, up.bias, down.bias]
    if len(eps) > 1:
        return None
    return (0, E, E * cfg.mlp_ratio, H, H, cfg.vocab_size, eps.pop()), found, _METHODS


class GPT2(nn.Module):
    def __init__(self, config):
        super().__init__()
        self.config = config
        self.embeddings = Embeddings(config)
        self.blocks = nn.ModuleList([TransformerBlock(config) for _ in range(config.num_blocks)])
        self.final_layer_norm = nn.LayerNorm(config.embed_dim, weight=config.use_layernorm_weight)
        self.lm_head = nn.Linear(config.embed_dim, config.vocab_size, bias=config.use_bias)
        self.apply(_init_weights)
        for name, param in self.named_parameters():
            if "out_proj" in name:
                nn.init.normal_(param, mean=0.0, std=0.02 / np.sqrt(2 * config.num_blocks))
        self.lm_head.weight = self.embeddings.char_embeddings.weight      # weight tying (:340-347)
        self._gradient_checkpointing_enabled = False

    def enable_gradient_checkpointing(self):
        """Recompute every transformer block in the backward pass instead of keeping its
        activations (gpt2.py:349-365)."""
        self._gradient_checkpointing_enabled = True

    def _planned(self, plan, ids, cache=None, last_only=False):
        """The whole forward as one library call (no graph); None when the cache is not as this model
        would have made it."""
        B, T = ids.shape
        past = cache.get_seq_len() if cache is not None else 0
        assert past + T <= (min(plan.positions, self.config.max_seq_len) if past else plan.positions), "position table exhausted"
        if cache is None:
            return plan.run(ids, last_only=last_only)
        cfg, n = self.config, cache.max_seq_len
        D = plan.head_dim
        if T > n or (past and D not in (64, 128)) or not cache.reserve(plan.blocks, B, cfg.num_heads, D, plan.dtype):
            return None
        L = len(cache.key_cache)
        ptrs = C.c_void_p * L
        out = plan.run(ids, past=past, position=past, write_pos=cache._appended[0] % n, kv_len=min(past + T, n), max_len=n,
                       k_cache=C.cast(ptrs(*[k.ptr for k in cache.key_cache]), C.c_void_p),
                       v_cache=C.cast(ptrs(*[v.ptr for v in cache.value_cache]), C.c_void_p),
                       cache_strides=_lib.Strides3(cfg.num_heads * n * D, n * D, D), last_only=last_only)
        cache._appended = [a + T for a in cache._appended]
        return out

    def forward(self, x, cache=None):
        """Logits; with a `Cache`, (logits, cache) as in gpt2.py:352-374."""
        from .utils.checkpoint import checkpoint
        plan = infer.plan_of(self, _plan)
        ids = infer.token_ids(x) if plan is not None else None
        if ids is not None:
            out = self._planned(plan, ids, cache)
            if out is not None:
                return Tensor(out) if cache is None else (Tensor(out), cache)
        past_length = cache.get_seq_len() if cache is not None else 0
        x = self.embeddings(x, past_length)
        for layer_idx, block in enumerate(self.blocks):
            if cache is not None:
                x = block(x, cache=cache, layer_idx=layer_idx)
            elif self._gradient_checkpointing_enabled and self.training and x.requires_grad:
                x = checkpoint(block, x)
            else:
                x = block(x)
        x = self.final_layer_norm(x)
        logits = self.lm_head(x)
        return logits if cache is None else (logits, cache)

    def _next_logits(self, feed, cache):
        """Logits [B, 1 or T, V] after the ids `feed`; the last position is the next token's."""
        plan = infer.plan_of(self, _plan)
        out = self._planned(plan, feed, cache, last_only=True) if plan is not None and feed.size else None
        if out is None:
            out = self.forward(Tensor(feed), cache=cache)
            out = (out if cache is None else out[0]).data
        return out

    def generate(self, input_ids, max_new_tokens, temperature=1.0, top_k=None, use_cache=True, seed=None):
        """Autoregressive sampling as in gpt2_trainer/inference_gpt2.py:137-174: the prompt fills
        the cache, then one token per step; temperature-scaled softmax (optionally restricted to
        the top_k logits), one draw per sequence on the host; temperature 0 takes the arg-max."""
        from .tensor import no_grad
        rng = np.random.default_rng(seed)
        ids = np.asarray(input_ids.numpy() if isinstance(input_ids, Tensor) else input_ids, dtype=np.int32)
        cache = Cache(self.config) if use_cache else None
        feed = ids
        with no_grad():
            if temperature == 0 and use_cache and max_new_tokens > 0 and ids.size and infer.plan_of(self, _plan) is not None:
                return infer.generate_greedy(self, ids, cache, max_new_tokens)
            for _ in range(max_new_tokens):
                logits = self._next_logits(Tensor(feed).data, cache)
                last = logits.numpy()[:, -1, :].astype(np.float64)
                if temperature == 0:
                    nxt = last.argmax(-1)
                else:
                    last = last / temperature
                    if top_k is not None:
                        kth = np.sort(last, -1)[:, -top_k][:, None]
                        last = np.where(last < kth, -np.inf, last)
                    p = np.exp(last - last.max(-1, keepdims=True))
                    p /= p.sum(-1, keepdims=True)
                    nxt = np.array([rng.choice(p.shape[-1], p=row) for row in p])
                ids = np.concatenate([ids, nxt[:, None].astype(np.int32)], axis=1)
                feed = ids[:, -1:] if use_cache else ids[:, -self.config.max_seq_len:]
        return ids


_METHODS = infer.methods(GPT2, Embeddings, TransformerBlock, Attention, FeedForward, nn.Linear, nn.LayerNorm, nn.Dropout)
