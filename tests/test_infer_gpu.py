"""The whole-model forward (mt_gpt_forward), the few-row products under it and the device arg-max,
against the op-by-op path of the same models and NumPy."""
import os
import subprocess
import sys

import numpy as np
import pytest

from tests.test_ops_gpu import DTYPES, TOL, close, dev, no_device_flag, rnd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mt():
    import mytorch_b200 as m
    return m


# One row up to the 64 the kernel takes and one beyond, both sides of the 16- and 32-row tiles; K with a
# ragged last step (40, 1000), split over 2, 4 and 8 blocks (1024, 2056, 4104); N with a partial group.
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,N,K", [(1, 8, 8), (1, 50257, 64), (2, 13, 40), (3, 776, 1000), (4, 64, 1024), (8, 768, 2056),
                                   (9, 100, 4104), (16, 2304, 768), (17, 33, 768), (32, 1280, 2048), (33, 72, 96), (64, 520, 776),
                                   (65, 72, 96)])
def test_few_row_products(mt, dtype, M, N, K):
    F = mt.fused_ops
    r = np.random.default_rng(M * 1000 + N)
    a, w = rnd(r.standard_normal((M, K)), dtype), rnd(r.standard_normal((N, K)) / np.sqrt(K), dtype)
    bias, res = rnd(r.standard_normal(N), dtype), rnd(r.standard_normal((M, N)), dtype)
    A, W, B, R = (dev(mt, v, dtype) for v in (a, w, bias, res))
    want = a.astype(np.float64) @ w.T.astype(np.float64)
    close(F.gemm(A, W, trans_b=True).numpy(), want, TOL[dtype], "plain")
    close(F.gemm(A, W, trans_b=True, bias=B, aux=R, aux_mode=1).numpy(), want + bias + res, TOL[dtype], "bias + residual")
    y = np.maximum(want + bias, 0)
    close(F.gemm(A, W, trans_b=True, bias=B, act="relu_squared").numpy(), y * y, 2 * TOL[dtype], "relu^2")
    no_device_flag(mt)


@pytest.mark.parametrize("dtype", DTYPES)
def test_argmax_rows(mt, dtype):
    from mytorch_b200 import _lib
    from mytorch_b200.array import DeviceArray, stream
    r = np.random.default_rng(1)
    for rows, cols in ((1, 1), (3, 7), (2, 50257), (5, 4096)):
        x = rnd(r.standard_normal((rows, cols)), dtype)
        x[:, cols // 2] = x[:, -1] = x.max(-1)                       # equals: the first one counts
        if rows > 2:
            x[1, cols // 3] = np.nan
        X, idx, out = dev(mt, x, dtype), DeviceArray.empty((rows,), "int32"), DeviceArray.zeros((rows, 4), "int32")
        _lib.argmax_rows(X.ptr, idx.ptr, out.ptr + 8, rows, cols, 4, X.code, stream())
        want = x.argmax(-1)
        assert np.array_equal(idx.numpy(), want) and np.array_equal(out.numpy()[:, 2], want)


def models(mt, kind, dtype, heads, kv_heads, D, bias):
    r = np.random.default_rng(3)
    if kind == "gpt2":
        from mytorch_b200.gpt2 import GPT2, GPT2Config
        model = GPT2(GPT2Config(vocab_size=203, max_seq_len=160, embed_dim=heads * D, num_blocks=2, num_heads=heads, use_bias=bias))
    else:
        from mytorch_b200.nanochat_gpt import GPT, GPTConfig
        model = GPT(GPTConfig(vocab_size=200, max_seq_len=160, embed_dim=heads * D, num_blocks=2, num_q_heads=heads,
                              num_kv_heads=kv_heads, use_bias=bias))
    for _, p in model.named_parameters():
        p.data.set_from_numpy((r.standard_normal(p.shape) * (0.05 if len(p.shape) > 1 else 0.3) + (len(p.shape) < 2)).astype(np.float32))
        p.astype(dtype)
    model.eval()
    return model


def cache_of(mt, model, kind, B):
    if kind == "gpt2":
        from mytorch_b200.gpt2 import Cache
        return Cache(model.config)
    from mytorch_b200.nanochat_gpt import KVCache
    c = model.config
    return KVCache(B, c.num_kv_heads, c.max_seq_len, c.embed_dim // c.num_q_heads, c.num_blocks)


# Groups of 1, 2, 5 and 6 query heads per key/value head (6 takes two blocks), batches on both sides of
# the 32 rows of the one-token schedule, prompts that end inside and beyond one pass over the keys.
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kind,heads,kv_heads,D,B,T,bias", [("gpt2", 2, 2, 64, 3, 70, False), ("gpt2", 2, 2, 64, 1, 5, True),
                                                            ("gpt2", 1, 1, 128, 33, 9, False), ("nanochat", 5, 1, 128, 2, 130, False),
                                                            ("nanochat", 6, 1, 64, 1, 33, True), ("nanochat", 4, 2, 128, 17, 12, False)])
def test_whole_model_forward_matches_the_ops(mt, monkeypatch, dtype, kind, heads, kv_heads, D, B, T, bias):
    """Prompt, single tokens and several tokens at once: the same logits from one library call as from
    the layers one by one. Half types: the layers round at the same places, so only the order of fp32 sums
    and the rounding of a few intermediate values differ."""
    from mytorch_b200 import infer
    model = models(mt, kind, dtype, heads, kv_heads, D, bias)
    ids = np.random.default_rng(5).integers(0, 200, (B, T + 8)).astype(np.int32)
    pieces = [ids[:, :T]] + [ids[:, T + i:T + i + 1] for i in range(4)] + [ids[:, T + 4:T + 6], ids[:, T + 6:T + 7]]

    def run():
        with mt.no_grad():
            whole = model(mt.Tensor(ids[:, :T]))
            got = [(whole[0] if kind == "nanochat" else whole).numpy()]
            cache = cache_of(mt, model, kind, B)
            for p in pieces:
                out = model(mt.Tensor(p), cache=cache) if kind == "gpt2" else model(mt.Tensor(p), None, cache=cache)
                got.append(out[0].numpy())
        return got
    one_call = run()
    assert model._infer_plan.ok
    monkeypatch.setattr(infer, "plan_of", lambda m, b: None)
    for a, b in zip(one_call, run()):
        close(a, b, 2 * TOL[dtype], "logits")
    no_device_flag(mt)


# Wide rows behind a norm: sizes whose rows, weights and sums no launch of the folded product holds (they take the norm and
# the product one after the other), and the last that one holds.
@pytest.mark.parametrize("dtype,width,B", [("float16", 4096, 10), ("bfloat16", 4096, 12), ("float16", 8192, 1), ("float32", 4096, 5),
                                           ("float32", 8192, 1), ("float16", 4096, 4)])
def test_wide_norm_and_head(mt, monkeypatch, dtype, width, B):
    from mytorch_b200 import infer
    from mytorch_b200.gpt2 import GPT2, GPT2Config
    model = GPT2(GPT2Config(vocab_size=3000, max_seq_len=2, embed_dim=width, num_blocks=0, num_heads=width // 128))
    for p in model.parameters():
        p.astype(dtype)
    ids = mt.Tensor(np.arange(B, dtype=np.int32)[:, None])
    with mt.no_grad():
        got = model(ids).numpy()
        assert model._infer_plan.ok
        monkeypatch.setattr(infer, "plan_of", lambda m, b: None)
        close(got, model(ids).numpy(), 2 * TOL[dtype], "logits")
    no_device_flag(mt)


def test_forced_kernels_are_used(mt, monkeypatch):
    """mt_gemm_force_simt holds for the products inside the library call: bit for bit the layers' results."""
    from mytorch_b200 import infer
    model = models(mt, "gpt2", "float32", 2, 2, 64, True)
    x = mt.Tensor(np.arange(5, dtype=np.int32)[None])
    mt._lib.gemm_force_simt(1)
    try:
        with mt.no_grad():
            one_call = model(x).numpy()
            monkeypatch.setattr(infer, "plan_of", lambda m, b: None)
            assert np.array_equal(one_call, model(x).numpy())
    finally:
        mt._lib.gemm_force_simt(0)


# K up to the longest that goes there, split over a cluster of eight
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("M,N,K", [(1, 72, 32768), (9, 100, 12288), (33, 40, 8192)])
def test_few_rows_of_long_k(mt, dtype, M, N, K):
    r = np.random.default_rng(K)
    a, w = rnd(r.standard_normal((M, K)), dtype), rnd(r.standard_normal((N, K)) / np.sqrt(K), dtype)
    got = mt.fused_ops.gemm(dev(mt, a, dtype), dev(mt, w, dtype), trans_b=True).numpy()
    close(got, a.astype(np.float64) @ w.T.astype(np.float64), TOL[dtype])
    no_device_flag(mt)


def steps(mt, kind):
    """Logits of a prompt and of steps behind it: the five-kernel schedule."""
    model = models(mt, kind, "float16", 4, 2, 64, True)
    ids = np.random.default_rng(5).integers(0, 200, (3, 70)).astype(np.int32)
    cache, got = cache_of(mt, model, kind, 3), []
    with mt.no_grad():
        for p in [ids[:, :64]] + [ids[:, t:t + 1] for t in range(64, 70)]:
            out = model(mt.Tensor(p), cache=cache) if kind == "gpt2" else model(mt.Tensor(p), None, cache=cache)
            got.append(out[0].numpy()[:, -1])
    return np.stack(got)


@pytest.mark.parametrize("kind", ["gpt2", "nanochat"])
def test_steps_without_overlap_and_on_another_stream(mt, tmp_path, kind):
    """Kernels that start before their predecessor has ended read nothing that it writes: the same bits with the overlap
    off (MT_PDL=0, read once per process), and on a stream of the caller's."""
    import ctypes as C
    from mytorch_b200 import _lib, array
    want = steps(mt, kind)
    code = f"import mytorch_b200 as mt, numpy as np, tests.test_infer_gpu as t; np.save({str(tmp_path / 'x.npy')!r}, t.steps(mt, {kind!r}))"
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    child = subprocess.run([sys.executable, "-c", code], cwd=root, env=dict(os.environ, MT_PDL="0"), capture_output=True, text=True, timeout=300)
    assert child.returncode == 0, child.stderr[-2000:]
    assert np.array_equal(np.load(tmp_path / "x.npy"), want)
    mine, before = C.c_void_p(), array.stream()
    array.synchronize()
    _lib.stream_create(C.byref(mine))
    array.set_stream(mine)
    try:
        assert np.array_equal(steps(mt, kind), want)
        array.synchronize()
    finally:
        array.set_stream(before)
    _lib.stream_destroy(mine)


def test_plans_follow_the_weights(mt):
    """Replaced, cast or reloaded weights are used by the next forward."""
    model = models(mt, "gpt2", "float32", 2, 2, 64, False)
    x = mt.Tensor(np.arange(12, dtype=np.int32).reshape(2, 6))
    with mt.no_grad():
        first = model(x).numpy()
        model.blocks[0].attention.qkv_proj.weight = mt.Tensor(np.zeros((384, 128), np.float32), requires_grad=True)
        second = model(x).numpy()
        for p in model.parameters():
            p.astype("float16")
        third = model(x)
    assert np.abs(first - second).max() > 1e-3 and third.dtype == "float16"
    close(third.numpy(), second, 1e-2, "after the cast")
