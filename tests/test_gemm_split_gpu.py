"""The tensor-core GEMM for fp32 matrices (three bf16 planes per operand) and for half matrices that TMA
cannot address: against 64-bit products, every operand order, ragged tiles, K split over a cluster,
epilogues, and operands that are not finite."""
import numpy as np
import pytest

from tests.test_ops_gpu import TOL, close, dev, no_device_flag, rnd

pytestmark = pytest.mark.gpu

ORDERS = [(0, 1), (0, 0), (1, 0), (1, 1)]


@pytest.fixture(scope="module")
def mt():
    import mytorch_b200 as m
    return m


def product(a, b, ta, tb):
    a, b = (a.T if ta else a).astype(np.float64), (b.T if tb else b).astype(np.float64)
    return a @ b, np.abs(a) @ np.abs(b)


def bound(K):
    # of sum |a||b|: 24 products are added to an accumulator that may cut off instead of rounding (2^-23 each), K/64
    # sums are rounded (2^-24 each), planes and left-out products 2^-23 together
    return (24 * 2 + K / 64 + 2) * 2.0 ** -24


# (each large enough for this path) one tile and less, ragged in every direction, pitches of 4, 8, 12 and odd bytes; few tiles with K split over 2, 4 and
# 8 CTAs (512, 1000, 4096); more tiles than SMs
@pytest.mark.parametrize("ta,tb", ORDERS)
@pytest.mark.parametrize("M,N,K", [(128, 128, 512), (129, 65, 1001), (72, 2000, 512), (67, 131, 1000), (256, 264, 4096), (300, 77, 4099),
                                   (1700, 1666, 90), (1630, 1560, 100)])
def test_fp32_products(mt, ta, tb, M, N, K):
    r = np.random.default_rng(M + N + K)
    a = r.standard_normal((K, M) if ta else (M, K)).astype(np.float32)
    b = (r.standard_normal((N, K) if tb else (K, N)) * np.exp(r.standard_normal((1, 1)))).astype(np.float32)
    want, size = product(a, b, ta, tb)
    C = mt.fused_ops.gemm(dev(mt, a, "float32"), dev(mt, b, "float32"), trans_a=bool(ta), trans_b=bool(tb)).numpy()
    assert (np.abs(C - want) <= bound(K) * size).all(), (np.abs(C - want) / size).max() / bound(K)
    no_device_flag(mt)


@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("ta,tb", ORDERS)
@pytest.mark.parametrize("M,N,K", [(129, 65, 1001), (300, 77, 4099), (1700, 1665, 91), (128, 264, 501)])
def test_half_products_with_odd_pitches(mt, dtype, ta, tb, M, N, K):
    r = np.random.default_rng(M + N + K)
    a, b = rnd(r.standard_normal((K, M) if ta else (M, K)), dtype), rnd(r.standard_normal((N, K) if tb else (K, N)), dtype)
    want, size = product(a, b, ta, tb)
    A, B = dev(mt, a, dtype), dev(mt, b, dtype)
    close(mt.fused_ops.gemm(A, B, trans_a=bool(ta), trans_b=bool(tb)).numpy(), want, TOL[dtype], "half output")
    acc = mt.DeviceArray.from_numpy(np.ones((M, N), np.float32))
    mt.fused_ops.gemm(A, B, trans_a=bool(ta), trans_b=bool(tb), out=acc, accumulate=2)
    assert (np.abs(acc.numpy() - 1 - want) <= bound(K) * (size + 1)).all()
    no_device_flag(mt)


def errors(mt, A, B, want, out_dtype):
    """Relative errors (2-norm) of A B^T as dispatched and as a chain of fp32 FMAs."""
    out = []
    for simt in (0, 1):
        mt._lib.gemm_force_simt(simt)
        try:
            got = mt.fused_ops.gemm(A, B, trans_b=True, out_dtype=out_dtype).numpy().astype(np.float64)
        finally:
            mt._lib.gemm_force_simt(0)
        out.append(np.linalg.norm(got - want) / np.linalg.norm(want))
    return out


# both sides of every length that the sum stays in tensor memory, and of the shortest K that goes there
@pytest.mark.parametrize("dtype", ["float16", "bfloat16"])
@pytest.mark.parametrize("K", [91, 255, 257, 2047, 2049, 12287, 12289, 49151, 50257])
def test_half_sums_are_no_less_exact_than_an_fp32_chain(mt, dtype, K):
    """Values of one sign: what the tensor cores cut off adds up in one direction. (A half output adds its own rounding, in
    which the sums' difference shows as less than 1 %.)"""
    n = 1000 if K < 3000 else 200
    r = np.random.default_rng(K)
    a, b = rnd(r.random((n, K)), dtype), rnd(r.random((n, K)) / np.sqrt(K), dtype)
    A, B = dev(mt, a, dtype), dev(mt, b, dtype)
    want = a.astype(np.float64) @ b.T.astype(np.float64)
    fast, chain = errors(mt, A, B, want, "float32")
    assert fast <= chain, (fast, chain)
    fast, chain = errors(mt, A, B, want, dtype)
    assert fast <= 1.01 * chain, (fast, chain)
    no_device_flag(mt)


# Magnitudes down to fp32's subnormals, whose last bits are what is left of a value; both one CTA per tile and a cluster
@pytest.mark.parametrize("M,N,K", [(300, 260, 500), (130, 70, 2000), (2100, 1000, 64)])
@pytest.mark.parametrize("ea,eb", [(-100, 0), (-112, 0), (-118, 10), (-126, 20), (-135, 60), (-147, 90), (90, -100), (60, 10)])
def test_small_and_large_magnitudes(mt, M, N, K, ea, eb):
    r = np.random.default_rng(K + 200 - ea)
    a = (r.standard_normal((M, K)) * 2.0 ** ea).astype(np.float32)
    b = (r.standard_normal((N, K)) * 2.0 ** eb).astype(np.float32)
    want, size = product(a, b, 0, 1)
    got = mt.fused_ops.gemm(dev(mt, a, "float32"), dev(mt, b, "float32"), trans_b=True).numpy()
    assert (np.abs(got - want) <= bound(K) * size + 2.0 ** -149).all(), (np.abs(got - want) / size).max() / bound(K)
    no_device_flag(mt)


@pytest.mark.parametrize("M,N,K", [(300, 260, 500), (130, 70, 2000)])          # one CTA per tile, a cluster per tile
def test_epilogues_match_the_cuda_core_kernel(mt, M, N, K):
    F = mt.fused_ops
    r = np.random.default_rng(5)
    X, W, B = (dev(mt, v.astype(np.float32), "float32") for v in (r.standard_normal((M, K)), r.standard_normal((N, K)) / np.sqrt(K),
                                                                  r.standard_normal(N)))
    aux = dev(mt, r.standard_normal((M, N)).astype(np.float32), "float32")

    def outputs():
        out = []
        for act in ("gelu", "relu_squared", "relu", None):
            for pre in (True, "grad"):
                out += [v.numpy() for v in F.gemm(X, W, trans_b=True, bias=B, act=act, preact=pre)]
        out += [F.gemm(X, W, trans_b=True, bias=B, aux=aux, aux_mode=mode).numpy() for mode in range(1, 7)]
        c = dev(mt, aux.numpy(), "float32")
        out.append(F.gemm(X, W, trans_b=True, alpha=0.5, out=c, accumulate=1).numpy())
        out.append(F.gemm(X, W, trans_b=True, out_dtype="float16").numpy().astype(np.float32))
        return out
    got = outputs()
    mt._lib.gemm_force_simt(1)
    try:
        want = outputs()
    finally:
        mt._lib.gemm_force_simt(0)
    for i, (g, w) in enumerate(zip(got, want)):
        close(g, w, 1e-3 if i == len(got) - 1 else 1e-5, f"epilogue {i}")
    no_device_flag(mt)


@pytest.mark.parametrize("M,N,K", [(300, 260, 500), (130, 70, 2000)])
def test_values_that_are_not_finite_come_out_as_in_fp32(mt, M, N, K):
    r = np.random.default_rng(6)
    a, b = r.standard_normal((M, K)).astype(np.float32), r.standard_normal((N, K)).astype(np.float32)
    b[:, 3] = 1.0
    a[5, 3], a[7, 3], a[9, 3], a[11, 3] = np.inf, -np.inf, np.nan, 3.4e38      # the last rounds to infinity in bf16
    A, B = dev(mt, a, "float32"), dev(mt, b, "float32")
    got = mt.fused_ops.gemm(A, B, trans_b=True).numpy()
    mt._lib.gemm_force_simt(1)
    try:
        want = mt.fused_ops.gemm(A, B, trans_b=True).numpy()
    finally:
        mt._lib.gemm_force_simt(0)
    assert np.isposinf(got[5]).all() and np.isneginf(got[7]).all() and np.isnan(got[9]).all()
    assert np.array_equal(np.isfinite(got), np.isfinite(want))
    ok = np.isfinite(want)
    assert np.abs(got[ok] / want[ok] - 1)[np.abs(want[ok]) > 1e30].max() <= 1e-5
    rows = np.isfinite(a).all(1)
    exact, size = product(a[rows], b, 0, 1)
    assert (np.abs(got[rows] - exact) <= bound(K) * size)[np.isfinite(want[rows])].all()


# many pieces to make up: whole operands, single rows and columns, results above the planes' range; one CTA, a pair and a
# cluster per tile, several tiles per CTA, every operand order, and the outputs that read what was there
@pytest.mark.parametrize("ta,tb", ORDERS)
@pytest.mark.parametrize("M,N,K", [(300, 260, 500), (130, 70, 2000), (2600, 2500, 130), (40, 300, 4096)])
@pytest.mark.parametrize("where", ["all", "row", "column", "large"])
def test_pieces_left_out_are_made_up(mt, M, N, K, ta, tb, where):
    F = mt.fused_ops
    r = np.random.default_rng(7)
    a, b = r.standard_normal((M, K)).astype(np.float32), r.standard_normal((N, K)).astype(np.float32)
    if where == "all":
        a[:] = np.nan
    elif where == "row":
        a[M // 2, K - 1] = np.inf
    elif where == "column":
        b[N - 1, 0] = np.nan
    else:
        a[M // 3], b[N // 2] = a[M // 3] * np.float32(1e20), b[N // 2] * np.float32(1e15)
    A, B = dev(mt, np.ascontiguousarray(a.T) if ta else a, "float32"), dev(mt, b if tb else np.ascontiguousarray(b.T), "float32")
    aux, bias = dev(mt, r.standard_normal((M, N)).astype(np.float32), "float32"), dev(mt, r.standard_normal(N).astype(np.float32), "float32")

    def outputs():
        c = dev(mt, aux.numpy(), "float32")
        y, pre = F.gemm(A, B, trans_a=bool(ta), trans_b=bool(tb), bias=bias, act="gelu", preact=True)
        return [F.gemm(A, B, trans_a=bool(ta), trans_b=bool(tb)).numpy(), F.gemm(A, B, trans_a=bool(ta), trans_b=bool(tb), out=c, accumulate=1).numpy(),
                F.gemm(A, B, trans_a=bool(ta), trans_b=bool(tb), aux=aux, aux_mode=1).numpy(), y.numpy(), pre.numpy()]
    got = outputs()
    mt._lib.gemm_force_simt(1)
    try:
        want = outputs()
    finally:
        mt._lib.gemm_force_simt(0)
    size = np.abs(np.nan_to_num(a, posinf=0)).astype(np.float64) @ np.abs(np.nan_to_num(b)).T.astype(np.float64)
    for i, (g, w) in enumerate(zip(got, want)):
        assert np.array_equal(np.isnan(g), np.isnan(w)) and np.array_equal(np.isinf(g), np.isinf(w)), i
        ok = np.isfinite(w)
        # both sides' sums; bias, aux and old values of size one; GELU's slope of up to 1.13
        assert (np.abs(g.astype(np.float64) - w) <= (bound(K) + (K + 4) * 2.0 ** -24) * 1.2 * (size + 8))[ok].all(), i
    no_device_flag(mt)
