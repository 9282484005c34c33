"""Stores of tensor-core products of few rows, on both sides of the row count up to
which rows go straight to memory (64): whole and ragged 32-column blocks, padded and
misaligned C, memory past the rows untouched.  Sums below 2^24, so exact."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off,pad", [(0, 0), (0, 4), (0, 3), (1, 0)])
@pytest.mark.parametrize("m,n", [(33, 64), (48, 300), (63, 256), (64, 100), (64, 257), (65, 96), (33, 65600)])
@pytest.mark.parametrize("dtype", ["i8", "i16", "bf16"])
def test_store_rows(fg, dtype, m, n, off, pad):
    from ferray_b200 import _lib as L
    k = 96
    r = np.random.default_rng(m + n)
    a, b = r.integers(-9, 10, (m, k)), r.integers(-9, 10, (k, n))
    code, ct = {"i8": (L.FG_I8, np.int32), "i16": (L.FG_I16, np.int32), "bf16": (L.FG_BF16, np.float32)}[dtype]
    if dtype == "bf16":
        a, b = ((x.astype(np.float32).view(np.uint32) >> 16).astype(np.uint16) for x in (a, b))
    else:
        a, b = (x.astype(dtype.replace("i", "int")) for x in (a, b))
    wide = (lambda x: (x.astype(np.uint32) << 16).view(np.float32)) if dtype == "bf16" else (lambda x: x)
    exact = wide(a).astype(np.float64) @ wide(b).astype(np.float64)
    da, db = fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b)
    ldc = n + pad
    c0 = r.integers(-1000, 1000, off + (m + 1) * ldc).astype(ct)
    ctx = fg.default_context()
    dc = fg.DeviceArray.from_numpy(c0)
    fg.check(ctx._lib.fg_gemm(ctx.handle, code, 0, 0, m, n, k, None, da.ptr, k, db.ptr, n, None,
                              C.c_void_p(dc.ptr + off * 4), ldc, 0, None))
    ctx.sync()
    want = c0.copy()
    want[off:].reshape(m + 1, ldc)[:m, :n] = exact
    np.testing.assert_array_equal(dc.to_numpy(), want)
