"""Model forwards without a graph as one library call (`mt_gpt_forward`): the inference branches of
gpt2_trainer/gpt2.py:352-374 and nanochat_trainer/core/nanochat_gpt.py:301-340.

A `Plan` describes a model's weights to the library. It is kept on the model and checked on every
use: each weight it was built from must still be the module's parameter and hold the same device
array, so loading, casting or replacing weights makes a new plan. Models that the call does not
cover (subclassed modules, dropout, mixed dtypes) return no plan and run op by op.
"""
import ctypes as C

from . import _lib
from .array import DeviceArray, stream
from .tensor import Tensor

# norm1 w, b; norm2 w, b; q (or qkv), k, v, out, up, down weights; their biases
_NO_STRIDES = _lib.Strides3(0, 0, 0)


def plain(module, cls):
    """The module is exactly `cls` with the class's own forward."""
    return type(module) is cls and "forward" not in module.__dict__


def greedy(logits, ids_out, column):
    """Arg-max of every row of logits [B, 1, V] into ids_out[:, column] (int32 on the device) and as
    the next step's ids [B, 1]."""
    B, V = logits.shape[0], logits.shape[-1]
    nxt = DeviceArray.empty((B, 1), "int32")
    _lib.argmax_rows(logits.ptr, nxt.ptr, ids_out.ptr + 4 * column, B, V, ids_out.shape[1], logits.code, stream())
    return nxt


class Plan:
    def __init__(self, model, kind, modules, blocks, block_modules, heads, kv_heads, hidden, vocab, cos=None, sin=None):
        """modules: {"wte", "wpe", "lnf", "head"} -> module or None; block_modules: per block the
        modules in the order norm1, norm2, q, k, v, out, up, down (None = absent)."""
        self.ok = False
        self.blocks = list(blocks)
        self.checks = []
        self.keep = (cos, sin)

        def ptr(module, name):
            t = None if module is None else getattr(module, name, None)
            if module is not None:
                self.checks.append((module, name, t, None if t is None else t.data))
            return t

        def address(t):
            return None if t is None else t.data.ptr
        top = {k: (ptr(m, "weight"), ptr(m, "bias")) for k, m in modules.items()}
        rows = []
        for mods in block_modules:
            w = [ptr(m, "weight") for m in mods]
            b = [ptr(m, "bias") for m in mods]
            rows.append([w[0], b[0], w[1], b[1], *w[2:], *b[2:]])
        tensors = [t for pair in top.values() for t in pair if t is not None] + [t for r in rows for t in r if t is not None]
        dtypes = {t.dtype for t in tensors}
        eps = {m.eps for m in [modules.get("lnf")] + [m for mods in block_modules for m in mods[:2]] if m is not None}
        if len(dtypes) != 1 or len(eps) > 1:
            return
        self.dtype = dtypes.pop()
        flat = [address(t) for r in rows for t in r]
        self.ptrs = (C.c_void_p * max(1, len(flat)))(*flat)
        wte = top["wte"][0]
        head_w, head_b = top["head"]
        width = wte.shape[1]
        self.c = _lib.GptModel(kind, wte.data.code, len(rows), width, hidden, heads, kv_heads, vocab, address(wte),
                               address(top["wpe"][0]) if "wpe" in top else None, *(map(address, top["lnf"]) if "lnf" in top else (None, None)),
                               address(head_w), address(head_b), None if cos is None else cos.ptr, None if sin is None else sin.ptr,
                               C.cast(self.ptrs, C.c_void_p), eps.pop() if eps else 1e-5)
        self.vocab, self.head_dim = vocab, width // heads
        D = self.head_dim
        q_rows = 3 * width if kind == 0 else heads * D
        want = [(width,)] * 4 + [(q_rows, width)] + [(kv_heads * D, width)] * 2 + [(width, heads * D), (hidden, width), (width, hidden)]
        shapes_ok = head_w.shape == (vocab, width) and all(t is None or t.shape == w for r in rows for t, w in zip(r, want))
        self.ok = shapes_ok and D <= 128

    def valid(self, blocks):
        if len(blocks) != len(self.blocks) or any(a is not b for a, b in zip(blocks, self.blocks)):
            return False
        for module, name, t, data in self.checks:
            now = getattr(module, name, None)
            if now is not t or (t is not None and t.data is not data):
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


def plan_of(model, build):
    """The model's plan, or None when a graph is being recorded, calls are traced one by one, or the
    model is outside what the call covers. `build(model)` makes a new one."""
    if Tensor.build_graph_enabled() or _lib._TRACE:
        return None
    plan = model.__dict__.get("_infer_plan")
    if plan is None or not plan.valid(model.blocks):
        plan = build(model)
        object.__setattr__(model, "_infer_plan", plan)
    return plan if plan.ok else None


class NoPlan:
    """Marks a model that the library call does not cover; looked at again when its blocks change."""
    ok = False

    def __init__(self, blocks):
        self.blocks = list(blocks)

    def valid(self, blocks):
        return len(blocks) == len(self.blocks) and all(a is b for a, b in zip(blocks, self.blocks))
