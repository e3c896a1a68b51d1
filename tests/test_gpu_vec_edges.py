"""BLAS-1 on device vectors at the edges of its forms: the integer conversions
between float and double (subnormal, zero of both signs, infinite, NaN, ties,
results that overflow or turn subnormal), 16-byte and unaligned pointers,
lengths around four.

Elementwise results are the bits of numpy's own conversions (the factors are
exact in double, so no rounding hides in the products).  The dot product adds
n products exactly representable in double, each addition rounding to 2^-53 of
a sum below sum |a b|: |error| <= n 2^-53 sum |a b|."""
import ctypes as C
import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

SPECIAL = np.array([0.0, -0.0, 1e-45, -1e-45, 1.1754942e-38, 1.17549435e-38, -1.17549435e-38, 3.4028235e38,
                    -3.4028235e38, np.inf, -np.inf, np.nan, 1.0, -1.0, 1.0000001, 16777217.0, 0.1, 3e-39],
                   np.float32)


def _lib():
    from sep_code_gb300 import gpu_funcs as gf
    from sep_code_gb300._lib import lib
    gf.setup_cuda(1)
    vp, ll, d = C.c_void_p, C.c_longlong, C.c_double
    lib.sepx_vec_scale.argtypes = [vp, ll, d]
    lib.sepx_vec_scale_add.argtypes = [vp, vp, ll, d, d]
    lib.sepx_vec_scale_add2.argtypes = [vp, vp, vp, ll, d, d]
    lib.sepx_vec_fill.argtypes = [vp, ll, C.c_float]
    for n in ("add", "mult"):
        getattr(lib, "sepx_vec_" + n).argtypes = [vp, vp, ll]
    return lib


def _same(a, b):
    return np.array_equal(a.view(np.uint32)[~np.isnan(a)], b.view(np.uint32)[~np.isnan(b)]) and \
        np.array_equal(np.isnan(a), np.isnan(b))


@pytest.mark.parametrize("n,off", [(1, 0), (3, 0), (4, 0), (5, 1), (1023, 0), (4 * len(SPECIAL) + 2, 0), (70001, 3)])
def test_elementwise_and_dot(n, off):
    lib = _lib()
    rng = np.random.default_rng(n)
    x1 = (rng.standard_normal(n) * np.exp(rng.uniform(-85, 80, n))).astype(np.float32)
    x2 = rng.standard_normal(n).astype(np.float32)
    k = min(n, len(SPECIAL))
    x1[:k] = SPECIAL[:k]
    buf = {s: torch.zeros(n + 8, dtype=torch.float32, device="cuda") for s in ("y", "a", "b")}
    y, a, b = (buf[s][off:off + n] for s in ("y", "a", "b"))
    p = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731

    def put(t, v):
        t.copy_(torch.tensor(v))
        torch.cuda.synchronize()

    def out(t):
        assert lib.sepx_synchronize() == 0
        return t.cpu().numpy()
    put(a, x1)
    put(b, x2)
    with np.errstate(all="ignore"):
        d1, d2 = x1.astype(np.float64), x2.astype(np.float64)
        # ties and range ends: x 1.5 of odd mantissas, / 2^126 into the subnormals, x 2^100 into infinity
        for f in (1.5, 2.0 ** -126, 2.0 ** 100, 1.0 + 2.0 ** -24):
            put(y, x1)
            assert lib.sepx_vec_scale(p(y), n, f) == 0
            assert _same(out(y), (d1 * f).astype(np.float32)), f
        assert lib.sepx_vec_scale_add2(p(y), p(a), p(b), n, 0.75, 0.0) == 0
        assert _same(out(y), (d1 * 0.75 + d2 * 0.0).astype(np.float32))
        put(y, x2)
        assert lib.sepx_vec_scale_add(p(y), p(b), n, 0.5, 2.0) == 0
        assert _same(out(y), (d2 * 0.5 + 2.0 * d2).astype(np.float32))
        put(y, x2)
        assert lib.sepx_vec_add(p(y), p(a), n) == 0
        assert _same(out(y), x2 + x1)
        put(y, x2)
        assert lib.sepx_vec_mult(p(y), p(a), n) == 0
        assert _same(out(y), x2 * x1)
    assert lib.sepx_vec_fill(p(y), n, -2.5) == 0
    assert (out(y) == -2.5).all() and (buf["y"].cpu().numpy()[off + n:] == 0).all()
    # dot: finite values
    fin = np.where(np.isfinite(x1) & (np.abs(x1) < 1e30), x1, 1.0).astype(np.float32)
    put(a, fin)
    r = C.c_double()
    for other, v in ((b, d2), (None, np.ones(n))):
        got = []
        for _ in range(2):
            assert lib.sepx_dot_f32(p(a), p(other) if other is not None else None, n, C.byref(r)) == 0
            got.append(r.value)
        prod = fin.astype(np.float64) * v
        assert abs(got[0] - math.fsum(prod)) <= n * 2.0 ** -53 * math.fsum(np.abs(prod)) + 5e-324
        assert got[0] == got[1]
