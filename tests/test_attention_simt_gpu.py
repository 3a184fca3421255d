"""The CUDA-core attention kernels (fp32, and half types at head sizes the tensor-core kernels do not take)
against a 64-bit computation: every padded head size, rows that no tile divides, both block heights,
grouped heads, strides and addresses that rule vector loads out."""
import numpy as np
import pytest

from tests.test_ops_gpu import TOL, close, dev, rnd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mt():
    import mytorch_b200 as m
    return m


def reference(q, k, v, d_o, causal):
    q, k, v, d_o = (a.astype(np.float64) for a in (q, k, v, d_o))
    g, S = q.shape[1] // k.shape[1], q.shape[2]
    scale = 1 / np.sqrt(q.shape[3])
    kk, vv = (np.repeat(a, g, 1) for a in (k, v))
    s = q @ kk.swapaxes(-1, -2) * scale
    if causal:
        s = np.where(np.tril(np.ones((S, S), bool)), s, -np.inf)
    m = s.max(-1, keepdims=True)
    p = np.exp(s - m)
    l = p.sum(-1, keepdims=True)
    p /= l
    o = p @ vv
    dp = d_o @ vv.swapaxes(-1, -2)
    ds = p * (dp - (d_o * o).sum(-1, keepdims=True)) * scale
    fold = lambda a: a.reshape(a.shape[0], -1, g, S, a.shape[3]).sum(2)
    return o, (m + np.log(l))[..., 0], ds @ kk, fold(ds.swapaxes(-1, -2) @ q), fold(p.swapaxes(-1, -2) @ d_o)


# sizes around the 64- and 128-row blocks; seven sequences of 16 heads take the 128-row block on 148 SMs
CASES = [("float32", 1, 2, 2, 3, 32), ("float32", 2, 4, 2, 63, 20), ("float32", 1, 2, 1, 64, 64), ("float32", 2, 3, 3, 65, 96),
         ("float32", 1, 4, 4, 129, 128), ("float32", 1, 2, 2, 200, 33), ("float32", 7, 16, 4, 300, 64), ("float32", 7, 16, 16, 301, 36),
         ("float32", 7, 16, 8, 257, 128), ("float32", 7, 16, 16, 260, 90), ("float16", 2, 4, 1, 130, 96), ("bfloat16", 7, 16, 16, 270, 32),
         ("float16", 1, 2, 2, 77, 31)]


@pytest.mark.parametrize("causal", [False, True])
@pytest.mark.parametrize("dtype,B,H,Hk,S,D", CASES)
def test_attention_matches_64_bits(mt, dtype, B, H, Hk, S, D, causal):
    F = mt.fused_ops
    r = np.random.default_rng(S + D)
    q, k, v, d_o = (rnd(r.standard_normal((B, h, S, D)), dtype) for h in (H, Hk, Hk, H))
    want = reference(q, k, v, d_o, causal)
    Q, K, V, G = (dev(mt, a, dtype) for a in (q, k, v, d_o))
    Q, K, V, o, lse = F.fused_sdpa_forward(Q, K, V, causal=causal)
    got = (o, lse) + tuple(F.fused_sdpa_backward(G, Q, K, V, o, lse, causal=causal))
    # fp32: the hardware exp2 (2^-22) of arguments up to ~10 that were rounded to 2^-24, twice in dS
    tol = 2e-5 if dtype == "float32" else TOL[dtype]
    for g, w, name in zip(got, want, ("o", "lse", "dq", "dk", "dv")):
        close(g.numpy(), w, tol, f"{name} {dtype} {B}x{H}/{Hk}x{S}x{D} causal={causal}")


@pytest.mark.parametrize("offset,row", [(0, 3 * 64 + 1), (1, 3 * 64), (4, 3 * 64 + 4)])
def test_strided_rows_in_one_buffer(mt, offset, row):
    """q, k and v side by side in rows of one buffer whose pitch or start may rule 16-byte loads out."""
    from mytorch_b200 import _lib
    from mytorch_b200.array import stream
    B, S, D = 2, 100, 64
    r = np.random.default_rng(0)
    x = r.standard_normal((B, S, row)).astype(np.float32)
    d_o = r.standard_normal((B, 1, S, D)).astype(np.float32)
    q, k, v = (x[:, None, :, i * D:(i + 1) * D] for i in range(3))
    want = reference(q, k, v, d_o, True)
    flat = np.concatenate([np.zeros(offset, np.float32), x.reshape(-1)])
    X, G = dev(mt, flat, "float32"), dev(mt, d_o, "float32")
    O, L = mt.DeviceArray.zeros((B, 1, S, D), "float32"), mt.DeviceArray.zeros((B, 1, S), "float32")
    st = _lib.Strides3
    sx, so = st(S * row, 0, row), st(S * D, S * D, D)
    ptr = [X.ptr + 4 * (offset + i * D) for i in range(3)]
    _lib.attn_fwd(*ptr, O.ptr, L.ptr, sx, sx, sx, so, B, 1, S, D, D ** -0.5, 1, X.code, stream())
    grads = [mt.DeviceArray.zeros((B, 1, S, D), "float32") for _ in range(3)]
    delta = mt.DeviceArray.zeros((B, 1, S), "float32")
    _lib.attn_bwd(*ptr, O.ptr, G.ptr, L.ptr, *(g.ptr for g in grads), delta.ptr, None, sx, sx, sx, so, so, so, so, so, B, 1, S, D,
                  D ** -0.5, 1, X.code, stream())
    for g, w, name in zip([O, L] + grads, want, ("o", "lse", "dq", "dk", "dv")):
        close(g.numpy(), w, 2e-5, name)


# a row in the first, a middle and the last of the 64-row tiles; both block heights, grouped heads, every padded head size
@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("dtype,B,H,Hk,S,D,t", [("float32", 1, 2, 1, 200, 64, 70), ("float32", 7, 16, 16, 260, 64, 127), ("float32", 1, 2, 2, 130, 32, 63),
                                                ("float32", 7, 16, 8, 257, 128, 200), ("float32", 1, 4, 4, 129, 90, 128), ("float16", 1, 2, 2, 140, 96, 3)])
def test_masked_values_that_are_not_finite_reach_no_row(mt, dtype, B, H, Hk, S, D, t, bad):
    """Row t of one operand is not finite: causal attention gives the rows that do not see it what it gives without it."""
    F = mt.fused_ops
    r = np.random.default_rng(S + D)
    clean = [rnd(r.standard_normal((B, h, S, D)), dtype) for h in (H, Hk, Hk, H)]
    want = reference(*clean, True)
    tol = 2e-5 if dtype == "float32" else TOL[dtype]

    def run(which):
        arrays = [a.copy() for a in clean]
        if which is not None:
            arrays[which][:, :, t, ::3] = bad
        Q, K, V, G = (dev(mt, a, dtype) for a in arrays)
        Q, K, V, o, lse = F.fused_sdpa_forward(Q, K, V, causal=True)
        return [a.numpy() for a in (o, lse) + tuple(F.fused_sdpa_backward(G, Q, K, V, o, lse, causal=True))]
    before, after = slice(0, t), slice(t + 1, S)
    # operand -> what does not depend on its row t: rows of o, lse and dq before a key's, of dk and dv behind a query's
    for which, parts in ((0, {0: before, 1: before, 2: before, 3: after, 4: after}), (1, {0: before, 1: before, 2: before}),
                         (2, {0: before, 2: before}), (3, {2: before, 3: after, 4: after})):
        got = run(which)
        for i, rows in parts.items():
            if rows.start < rows.stop:
                close(got[i][:, :, rows], want[i][:, :, rows], tol, f"operand {which}, result {i}")
        if which == 2:
            assert not np.isfinite(got[0][:, :, t, ::3]).any()
