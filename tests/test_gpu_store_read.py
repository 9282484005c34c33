"""Tensor-core products that read C: row counts around the 4-, 16- and 32-row steps
of the store, whole, ragged and misaligned column blocks, all epilogues.  Integer
values below 2^24, scale and beta powers of two, so every result is exact."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(fg, x):
    return fg.DeviceArray.from_numpy(np.ascontiguousarray(x))


@pytest.mark.parametrize("off,pad", [(0, 0), (0, 4), (1, 3)])
@pytest.mark.parametrize("m,n", [(1, 32), (15, 100), (17, 64), (31, 33), (48, 256), (67, 259), (130, 300), (257, 520)])
@pytest.mark.parametrize("dtype", ["i8", "i16", "bf16", "f32", "f32_3"])
def test_accumulate(fg, dtype, m, n, off, pad):
    from ferray_b200 import _lib as L
    k = 70
    r = np.random.default_rng(m + n)
    a, b = r.integers(-9, 10, (m, k)), r.integers(-9, 10, (k, n))
    exact = a.astype(np.float64) @ b
    code, mode, ct, slices, beta = {
        "i8": (L.FG_I8, 0, np.int32, 0, 1), "i16": (L.FG_I16, 0, np.int32, 0, 1), "bf16": (L.FG_BF16, 0, np.float32, 0, 1),
        "f32": (L.FG_F32, 1, np.float32, 2, -2), "f32_3": (L.FG_F32, 1, np.float32, 3, -2)}[dtype]
    if dtype == "bf16":
        a, b = ((x.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16) for x in (a, b))
    elif code == L.FG_F32:
        a, b = a.astype(np.float32), b.astype(np.float32)
    else:
        a, b = (x.astype(dtype.replace("i", "int")) for x in (a, b))
    one, be = (C.c_float * 1)(1.0), (C.c_float * 1)(beta)
    da, db = _dev(fg, a), _dev(fg, b)
    ldc = n + pad
    c0 = r.integers(-1000, 1000, off + (m + 1) * ldc).astype(ct)
    dc = _dev(fg, c0)
    ctx = fg.default_context()
    f32 = code == L.FG_F32
    fg.check(ctx._lib.fg_gemm(ctx.handle, code, mode, slices, m, n, k, one if f32 else None, da.ptr, k, db.ptr, n,
                              be if f32 else None, C.c_void_p(dc.ptr + off * 4), ldc, 0 if f32 else 1, None))
    ctx.sync()
    want = c0.copy()
    rows = want[off:].reshape(m + 1, ldc)[:m, :n]
    rows[:] = rows * beta + exact
    np.testing.assert_array_equal(dc.to_numpy(), want)


@pytest.mark.parametrize("m,n", [(1, 32), (17, 33), (67, 259), (130, 256), (300, 520)])
def test_quantized_accumulate(fg, m, n):
    k = 70
    r = np.random.default_rng(m + n)
    a, b = r.integers(0, 30, (m, k), dtype=np.uint8), r.integers(-20, 20, (k, n), dtype=np.int8)
    c0 = r.integers(-1000, 1000, (m, n)).astype(np.float32)
    dc = _dev(fg, c0)
    assert fg.quantized_matmul(m, n, k, _dev(fg, a), 3, 0.5, _dev(fg, b), -2, 0.25, dc, accumulate=True)
    want = c0 + 0.125 * ((a.astype(np.int64) - 3) @ (b.astype(np.int64) + 2))
    np.testing.assert_array_equal(dc.to_numpy(), want)
