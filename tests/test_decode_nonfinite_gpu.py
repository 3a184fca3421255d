"""Decode attention with cached rows that are not finite: what depends on them is NaN, whichever lanes, warps or blocks
read them, and nothing else is touched."""
import numpy as np
import pytest

from tests.test_ops_gpu import DTYPES, TOL, close, dev, rnd

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mt():
    import mytorch_b200 as m
    return m


# one key, less than a warp's pass, a split over several blocks; one query head per key/value head and groups of 5 and 6
@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("kv_heads,group,n,D,at", [(2, 1, 1, 64, 0), (2, 1, 7, 64, 6), (2, 5, 40, 128, 39), (1, 6, 300, 64, 150),
                                                   (2, 1, 1000, 128, 999)])
def test_a_nan_key_or_value(mt, dtype, kv_heads, group, n, D, at):
    from mytorch_b200 import _lib
    from mytorch_b200.array import stream
    r = np.random.default_rng(n)
    B, H, rows = 2, kv_heads * group, n + 3
    q, k, v = (rnd(r.standard_normal((B, h, m, D)), dtype) for h, m in ((H, 1), (kv_heads, rows), (kv_heads, rows)))
    kk, vv = (np.repeat(a[:, :, :n], group, 1).astype(np.float64) for a in (k, v))
    s = q @ kk.swapaxes(-1, -2) * D ** -0.5
    p = np.exp(s - s.max(-1, keepdims=True))
    want = p / p.sum(-1, keepdims=True) @ vv
    st = _lib.Strides3

    def run(k, v):
        Q, K, V, O = dev(mt, q, dtype), dev(mt, k, dtype), dev(mt, v, dtype), dev(mt, np.zeros((B, H, 1, D)), dtype)
        sq, sc = st(H * D, D, D), st(kv_heads * rows * D, rows * D, D)
        _lib.attn_decode_gqa(Q.ptr, K.ptr, V.ptr, O.ptr, sq, sc, sq, B, H, kv_heads, 1, n, D, D ** -0.5, -1, Q.code, stream())
        return O.numpy()
    k[:, :, n:] = v[:, :, n:] = np.nan                   # rows past the cache's length are not read
    close(run(k, v), want, 2 * TOL[dtype], "finite")
    bad = k.copy()
    bad[1, kv_heads - 1, at, D // 2] = np.nan
    got = run(bad, v)
    hit = np.zeros((B, H), bool)
    hit[1, H - group:] = True
    assert np.isnan(got[hit]).all()
    close(got[~hit], want[~hit], 2 * TOL[dtype], "other heads, NaN key")
    bad = v.copy()
    bad[1, kv_heads - 1, at, 3] = np.nan
    got = run(k, bad)
    assert np.isnan(got[1, H - group:, 0, 3]).all() and np.isnan(got).sum() == group
