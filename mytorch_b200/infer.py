"""Model forwards without a graph as one library call (`mt_gpt_forward`): the inference branches of
gpt2_trainer/gpt2.py:352-374 and nanochat_trainer/core/nanochat_gpt.py:301-340.

A `Plan` describes a model's weights to the library: addresses and sizes. It is kept on the model and
looked over by every forward: no module has had an attribute assigned since, the sizes in the config, the blocks and
the classes' forwards are the same, and every weight still holds the same array. Otherwise the model is
walked and described anew, so replaced modules, weights, tables and options take effect at once. The
plan holds weak references only, so it keeps no array of the model alive. Models that the call does not
cover (subclassed or patched modules, dropout, other activations, mixed dtypes, tensors of unexpected
shapes) return no plan and run op by op. Looking a plan of 12 blocks over takes 10 us of host time, a
walk 50: a step of a small batch is bound by the host.
"""
import ctypes as C
import weakref

import numpy as np

from . import _lib
from .array import DeviceArray, code, stream
from .nn.modules import Module
from .tensor import Tensor

_NO_STRIDES = _lib.Strides3(0, 0, 0)
TOP, PER_BLOCK = 8, 16        # arrays of a description: the model's own, then each block's


def plain(module, cls):
    """The module is exactly `cls` with the class's own forward."""
    return module.__class__ is cls and "forward" not in module.__dict__


def methods(*classes):
    """The forwards (and Module.__call__) that the library call stands for, as they are at import."""
    return [(c, "forward", c.forward) for c in classes] + [(Module, "__call__", Module.__call__)]


def config_of(model):
    """What the descriptions read of a config, whatever kind of object that is."""
    c = model.config
    return [getattr(c, n, None) for n in ("embed_dim", "mlp_ratio", "vocab_size", "num_heads", "num_q_heads", "num_kv_heads")]


def unpatched(known):
    return all(getattr(c, name) is f for c, name, f in known)


def token_ids(x):
    """The ids [B, T] on the device; None for what the library call does not take (the layers then
    accept or refuse it)."""
    a = x.data if isinstance(x, Tensor) else DeviceArray.from_numpy(x, "int32")
    return a if a.dtype == "int32" and len(a.shape) == 2 and a.size else None


def greedy(logits, ids_out, column):
    """Arg-max of every sequence's last row of logits [B, T, V] into ids_out[:, column] (int32 on the
    device) and as the next step's ids [B, 1]."""
    B, T, V = logits.shape
    if T > 1:
        logits = DeviceArray.from_numpy(logits.numpy()[:, -1:, :], logits.dtype)
    nxt = DeviceArray.empty((B, 1), "int32")
    _lib.argmax_rows(logits.ptr, nxt.ptr, ids_out.ptr + 4 * column, B, V, ids_out.shape[1], logits.code, stream())
    return nxt


def generate_greedy(model, ids, cache, n):
    """[ids | n tokens]: the arg-max stays on the device and is the next step's input, so the host
    queues all steps and reads the tokens back once."""
    out, feed = DeviceArray.empty((ids.shape[0], n), "int32"), Tensor(ids).data
    for i in range(n):
        feed = greedy(model._next_logits(feed, cache), out, i)
    return np.concatenate([ids, out.numpy()], axis=1)


class Plan:
    """sizes: (kind, width, hidden, heads, kv_heads, vocab, eps); tensors: the token and position
    tables, the final norm's weight and bias, the head's weight and bias, the rotary tables (arrays),
    then per block 16 in the order of `block_ptrs` in mytorch_b200.h; None where there is none."""

    def __init__(self, model, edits, sizes, tensors, known):
        self.edits, self.config, self.known, self.ok = edits, config_of(model), known, False
        self.block_refs = [weakref.ref(b) for b in model.blocks]
        self.refs = [(weakref.ref(t), weakref.ref(t.data)) for t in tensors if isinstance(t, Tensor)]
        held = [t.data if isinstance(t, Tensor) else t for t in tensors]
        found = [None if a is None else (a.ptr, a.shape, a.dtype) for a in held]
        blocks = len(self.block_refs)
        kind, width, hidden, heads, kv_heads, vocab, eps = sizes
        self.blocks, self.vocab, self.head_dim = blocks, vocab, width // heads
        D = self.head_dim
        dtypes = {f[2] for i, f in enumerate(found) if f is not None and i not in (6, 7)}
        table = found[6] if kind else found[1]              # rotary tables; learned positions
        if len(dtypes) != 1 or D > 128 or table is None or found[0] is None or found[4] is None:
            return
        self.dtype = dtypes.pop()
        self.positions = table[1][0]
        pos = (self.positions, D if kind else width)
        q_rows, kv = heads * D if kind else 3 * width, kv_heads * D
        want = [(vocab, width), pos, (width,), (width,), (vocab, width), (vocab,), pos, pos]
        block = [(width,)] * 4 + [(q_rows, width), (kv, width), (kv, width), (width, heads * D), (hidden, width), (width, hidden),
                                  (q_rows,), (kv,), (kv,), (width,), (hidden,), (width,)]
        need = (4, 5, 6, 7, 8, 9) if kind else (4, 7, 8, 9)   # the projections
        rows = [found[TOP + PER_BLOCK * i:TOP + PER_BLOCK * (i + 1)] for i in range(blocks)]
        if any(f is not None and f[1] != w for f, w in zip(found, want)) or any(r[i] is None for r in rows for i in need) \
                or any(f is not None and f[1] != w for r in rows for f, w in zip(r, block)) \
                or (kind and any(f is None or f[2] != "float32" for f in found[6:8])):
            return
        ptr = [None if f is None else f[0] for f in found]
        self.ptrs = (C.c_void_p * max(1, len(ptr) - TOP))(*ptr[TOP:])
        self.c = _lib.GptModel(kind, code(self.dtype), blocks, width, hidden, heads, kv_heads, vocab, *ptr[:TOP],
                               C.cast(self.ptrs, C.c_void_p), eps)
        self.ok = True

    def current(self, model):
        if self.edits != Module.edits or config_of(model) != self.config or len(model.blocks) != len(self.block_refs) \
                or not unpatched(self.known):
            return False
        for b, r in zip(model.blocks, self.block_refs):
            if b is not r():
                return False
        for r, a in self.refs:
            t = r()
            if t is None or t.data is not a():
                return False
        return True

    def run(self, ids, past=0, position=0, write_pos=0, kv_len=0, max_len=0, k_cache=None, v_cache=None, cache_strides=None,
            last_only=False, softcap=0.0):
        """Logits [B, T, vocab] ([B, 1, vocab] with last_only)."""
        B, T = ids.shape
        logits = DeviceArray.empty((B, 1 if last_only else T, self.vocab), self.dtype)
        p = _lib.GptPass(ids.ptr, B, T, past, position, write_pos, kv_len, max_len, k_cache, v_cache,
                         cache_strides or _NO_STRIDES, logits.ptr, int(last_only), softcap)
        _lib.gpt_forward(C.byref(self.c), C.byref(p), stream())
        return logits


def plan_of(model, describe):
    """The model's plan as the model is now; None when a graph is being recorded, calls are traced one
    by one, or the model is outside what the call covers. `describe(model)` walks the model and
    returns (sizes, tensors, methods it stands for) as Plan takes them, or None."""
    if Tensor.build_graph_enabled() or _lib._TRACE:
        return None
    plan = model.__dict__.get("_infer_plan")
    if plan is None or not plan.current(model):
        edits = Module.edits                    # read before the walk: an edit during it makes the plan old
        found = describe(model)
        plan = None if found is None else Plan(model, edits, *found)
        object.__setattr__(model, "_infer_plan", plan)
    return plan if plan is not None and plan.ok else None
