"""Which weights, tables and options the whole-model forward (infer.plan_of) hands to the library, with device
arrays that are only addresses: everything that is replaced after a first forward has to be seen by the next one."""
import ctypes as C
import gc
import itertools
import weakref

import numpy as np
import pytest

import mytorch_b200 as mt
from mytorch_b200 import _lib, array, gpt2, infer, nanochat_gpt, nn
from mytorch_b200.array import DeviceArray


class Calls(list):
    """mt_gpt_forward as recorded: (sizes and addresses of the model, its blocks' addresses, the pass)."""

    def __call__(self, model, passed, stream):
        m, p = model._obj, passed._obj
        table = C.cast(m.block_ptrs, C.POINTER(C.c_void_p))
        self.append(({n: getattr(m, n) for n, _ in m._fields_ if n != "block_ptrs"}, [table[i] for i in range(16 * m.blocks)],
                     {n: getattr(p, n) for n, _ in p._fields_}))


@pytest.fixture
def calls(monkeypatch):
    address = itertools.count(4096, 4096)
    fake = lambda shape, dtype="float32": DeviceArray(next(address), shape, dtype)
    monkeypatch.setattr(DeviceArray, "empty", staticmethod(fake))
    monkeypatch.setattr(DeviceArray, "from_numpy", staticmethod(
        lambda a, dtype=None: fake(np.shape(a), dtype or ("int32" if np.asarray(a).dtype.kind == "i" else "float32"))))
    for name in ("set_from_numpy", "zero_", "fill_", "copy_from"):
        monkeypatch.setattr(DeviceArray, name, lambda self, *a: self)
    monkeypatch.setattr(array, "_stream", C.c_void_p(0))
    monkeypatch.setattr(_lib, "_TRACE", "")
    seen = Calls()
    monkeypatch.setattr(_lib, "gpt_forward", seen)
    return seen


def gpt2_model(**more):
    return gpt2.GPT2(gpt2.GPT2Config(vocab_size=96, max_seq_len=32, embed_dim=128, num_blocks=2, num_heads=2, **more))


def nano_model():
    m = nanochat_gpt.GPT(nanochat_gpt.GPTConfig(vocab_size=96, max_seq_len=32, embed_dim=128, num_blocks=2, num_q_heads=2, num_kv_heads=1))
    m.eval()
    return m


def weight(*shape):
    return nn.Linear(shape[1], shape[0], bias=False)


GPT2_EDITS = {
    "qkv projection": lambda m: setattr(m.blocks[1].attention, "qkv_proj", weight(384, 128)),
    "attention": lambda m: setattr(m.blocks[0], "attention", gpt2.Attention(m.config)),
    "feedforward": lambda m: setattr(m.blocks[1], "feedforward", gpt2.FeedForward(m.config)),
    "norm": lambda m: setattr(m.blocks[1], "layernorm2", nn.LayerNorm(128, bias=False)),
    "block": lambda m: m.blocks._list.__setitem__(1, gpt2.TransformerBlock(m.config)),
    "fewer blocks": lambda m: m.blocks._list.pop(),
    "head": lambda m: setattr(m, "lm_head", weight(96, 128)),
    "final norm": lambda m: setattr(m, "final_layer_norm", nn.LayerNorm(128)),
    "embeddings": lambda m: setattr(m, "embeddings", gpt2.Embeddings(m.config)),
    "positions": lambda m: setattr(m.embeddings, "position_embeddings", nn.Embedding(32, 128)),
    "eps": lambda m: [setattr(n, "eps", 1e-3) for b in m.blocks for n in (b.layernorm1, b.layernorm2)] + [setattr(m.final_layer_norm, "eps", 1e-3)],
    "weight": lambda m: setattr(m.blocks[0].feedforward.out_proj, "weight", weight(128, 512).weight),
    "weight's array": lambda m: setattr(m.blocks[0].feedforward.out_proj.weight, "data", DeviceArray.empty((128, 512))),
}
# what the library call does not cover: the layers have to run one by one
GPT2_OUTSIDE = {
    "own projection": lambda m: setattr(m.blocks[1].attention, "qkv_proj", type("Adapter", (nn.Linear,), {})(128, 384, bias=False)),
    "own head": lambda m: setattr(m, "lm_head", type("Head", (nn.Linear,), {})(128, 96, bias=False)),
    "one norm's eps": lambda m: setattr(m.blocks[0].layernorm1, "eps", 1e-3),
    "activation": lambda m: setattr(m.blocks[1].feedforward.intermediate_dense, "act_func", "relu"),
    "head's activation": lambda m: setattr(m.lm_head, "act_func", "gelu"),
    "dropout": lambda m: setattr(m.blocks[0].attention.proj_drop, "p", 0.1),
    "own forward": lambda m: setattr(m.blocks[1].feedforward, "forward", lambda x, residual=None: x),
    "one dtype": lambda m: setattr(m.lm_head.weight, "data", DeviceArray.empty((96, 128), "float16")),
    "short token table": lambda m: setattr(m.embeddings.char_embeddings.weight, "data", DeviceArray.empty((95, 128))),
    "narrow positions": lambda m: setattr(m.embeddings.position_embeddings.weight, "data", DeviceArray.empty((32, 64))),
    "final norm's size": lambda m: setattr(m.final_layer_norm.bias, "data", DeviceArray.empty((64,))),
    "bias's size": lambda m: setattr(m.blocks[0].attention.out_proj, "bias", mt.Tensor(DeviceArray.empty((64,)), requires_grad=True)),
    "heads": lambda m: setattr(m.blocks[0].attention, "num_heads", 1),
    "config": lambda m: setattr(m.config, "num_heads", 4),
    "own class": lambda m: setattr(m.blocks[0].attention, "__class__", type("Mine", (gpt2.Attention,), {})),
}
NANO_EDITS = {
    "key projection": lambda m: setattr(m.blocks[1].attention, "k_proj", weight(64, 128)),
    "head": lambda m: setattr(m, "lm_head", weight(96, 128)),
    "embeddings": lambda m: setattr(m.embeddings, "embeddings", nn.Embedding(96, 128)),
    "buffers": lambda m: m.register_buffer("cos", DeviceArray.empty((32, 64))),
    "rotary tables": lambda m: (setattr(m, "cos", DeviceArray.empty((32, 64))), setattr(m, "sin", DeviceArray.empty((32, 64)))),
}
NANO_OUTSIDE = {
    "activation": lambda m: setattr(m.blocks[1].feedforward.intermediate_dense, "act_func", "gelu"),
    "rotary tables' size": lambda m: setattr(m, "sin", DeviceArray.empty((32, 32))),
    "own forward": lambda m: setattr(m.blocks[1].attention, "forward", lambda x, *a, **k: x),
}


def forward(model, ids=None):
    with mt.no_grad():
        plan = infer.plan_of(model, gpt2._plan if isinstance(model, gpt2.GPT2) else nanochat_gpt._plan)
        return plan is not None and model._planned(plan, ids or DeviceArray.empty((2, 5), "int32"), None) is not None


def expected(model):
    """Addresses of the model's own arrays and of its blocks' projections and norms, as the model is now."""
    d = lambda t: None if t is None else t.data.ptr
    if isinstance(model, gpt2.GPT2):
        e, h, n = model.embeddings, model.lm_head, model.final_layer_norm
        top = dict(wte=d(e.char_embeddings.weight), wpe=d(e.position_embeddings.weight), head_w=d(h.weight), lnf_w=d(n.weight), lnf_b=d(n.bias))
        rows = [[d(b.layernorm1.weight), d(b.layernorm2.weight), d(b.attention.qkv_proj.weight), d(b.attention.out_proj.weight),
                 d(b.feedforward.intermediate_dense.weight), d(b.feedforward.out_proj.weight)] for b in model.blocks]
        return top, rows, (0, 2, 4, 7, 8, 9), model.final_layer_norm.eps
    top = dict(wte=d(model.embeddings.embeddings.weight), head_w=d(model.lm_head.weight), cos_t=model.cos.ptr, sin_t=model.sin.ptr)
    rows = [[d(m.weight) for m in (b.attention.q_proj, b.attention.k_proj, b.attention.v_proj, b.attention.out_proj,
                                   b.feedforward.intermediate_dense, b.feedforward.out_proj)] for b in model.blocks]
    return top, rows, (4, 5, 6, 7, 8, 9), 1e-5


@pytest.mark.parametrize("make,edit", [(gpt2_model, k) for k in GPT2_EDITS] + [(nano_model, k) for k in NANO_EDITS])
def test_what_is_replaced_is_used(calls, make, edit):
    model = make()
    assert forward(model)
    (GPT2_EDITS if make is gpt2_model else NANO_EDITS)[edit](model)
    assert forward(model)
    got, blocks, _ = calls[-1]
    top, rows, at, eps = expected(model)
    assert {k: got[k] for k in top} == top and got["blocks"] == len(rows) and got["eps"] == np.float32(eps)
    assert [[blocks[16 * i + j] for j in at] for i in range(len(rows))] == rows


@pytest.mark.parametrize("make,edit", [(gpt2_model, k) for k in GPT2_OUTSIDE] + [(nano_model, k) for k in NANO_OUTSIDE])
def test_what_the_call_does_not_cover_runs_op_by_op(calls, make, edit):
    model = make()
    assert forward(model)
    (GPT2_OUTSIDE if make is gpt2_model else NANO_OUTSIDE)[edit](model)
    assert not forward(model)


def test_patched_classes_run_op_by_op(calls, monkeypatch):
    model = gpt2_model()
    assert forward(model)
    monkeypatch.setattr(gpt2.Attention, "forward", lambda self, x, **k: x)
    assert not forward(model)


def test_configs_of_any_kind(calls):
    """Attributes in slots or on the class are read like a dataclass's."""
    plain = gpt2.GPT2Config(vocab_size=96, max_seq_len=32, embed_dim=128, num_blocks=2, num_heads=2)
    names = list(vars(plain))
    slots = type("Slots", (), {"__slots__": names})()
    for n in names:
        setattr(slots, n, getattr(plain, n))
    held = type("Held", (), dict(vars(plain)))
    for config, edit in ((slots, slots), (held(), held), (held, held)):
        model = gpt2.GPT2(config)
        assert forward(model) and forward(model)
        edit.num_heads = 4
        assert not forward(model)
        edit.num_heads = 2


def test_old_arrays_are_not_held(calls):
    model = gpt2_model()
    assert forward(model)
    old = [weakref.ref(p.data) for p in model.parameters()] + [weakref.ref(model.blocks[0].attention)]
    model.blocks[0].attention = gpt2.Attention(model.config)
    for p in model.parameters():
        p.data = DeviceArray.empty(p.shape, "float16")
    del p
    gc.collect()
    assert all(r() is None for r in old)


def test_a_plan_is_kept_while_nothing_changes(calls):
    model = gpt2_model()
    assert forward(model)
    plan = model._infer_plan
    model.train()
    model.eval()
    assert forward(model) and model._infer_plan is plan
    nn.Linear(1, 1).act_func = None           # any module's edit: looked at again
    assert forward(model) and model._infer_plan is not plan


@pytest.mark.parametrize("ids", [np.arange(10).reshape(2, 5), [[1, 2, 3]], np.arange(6, dtype=np.int32).reshape(1, 6)])
def test_ids_from_the_host(calls, ids):
    with mt.no_grad():
        gpt2_model()(ids)
        if not isinstance(ids, list):
            nano_model()(ids)
    assert len(calls) == (1 if isinstance(ids, list) else 2)
    assert all((p["batch"], p["new_tokens"]) == np.shape(ids) for _, _, p in calls)


def test_ids_of_other_kinds_go_to_the_layers(calls):
    assert infer.token_ids(mt.Tensor(DeviceArray.empty((2, 5), "int64"))) is None
    assert infer.token_ids(mt.Tensor(DeviceArray.empty((2, 0), "int32"))) is None
    assert infer.token_ids(mt.Tensor(DeviceArray.empty((5,), "int32"))) is None


def test_caches_of_another_shape_go_to_the_layers(calls):
    model = gpt2_model()
    ids = DeviceArray.empty((2, 5), "int32")
    plan = lambda: infer.plan_of(model, gpt2._plan)

    def cache(**more):
        return gpt2.Cache(gpt2.GPT2Config(**{**dict(max_seq_len=32, embed_dim=128, num_blocks=2, num_heads=2), **more}))
    with mt.no_grad():
        c = cache()
        assert model._planned(plan(), ids, c) is not None and c.get_seq_len(1) == 5
        assert model._planned(plan(), DeviceArray.empty((3, 1), "int32"), c) is None         # another batch
        c.value_cache[1] = DeviceArray.empty((2, 4, 32, 32))
        assert model._planned(plan(), ids, c) is None
        for n in (1, 3):                                                                     # the call reads one pointer per block
            c = cache(num_blocks=n)
            assert model._planned(plan(), ids, c) is None and c.key_cache == [None] * n
        assert model._planned(plan(), ids, cache(max_seq_len=4)) is None
        with pytest.raises(AssertionError, match="position table"):
            model._planned(plan(), DeviceArray.empty((1, 33), "int32"), None)
        nano = nano_model()
        k = nanochat_gpt.KVCache(2, 1, 32, 64, 2)
        k.k_cache = DeviceArray.empty((2, 2, 1, 16, 64))
        assert nano._planned(infer.plan_of(nano, nanochat_gpt._plan), ids, k) is None
