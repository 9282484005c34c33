"""Stores of the tensor-core products through shared memory, and the 256 x 256
tile of the 16-bit product: row and column counts around the 32-row blocks and
the 256-wide tiles, padded and misaligned C, with and without reading C.
Integer-valued operands whose sums stay below 2^24, so every result is exact."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bf16(x):
    return (np.ascontiguousarray(x, np.float32).view(np.uint32) >> 16).astype(np.uint16)  # exact for small integers


@pytest.mark.parametrize("off,pad", [(0, 0), (0, 4), (0, 3), (4, 4), (1, 1)])
@pytest.mark.parametrize("dtype,m,n,k", [
    (d, *s) for d in ("i8", "i16", "bf16")
    for s in [(1, 32, 64), (16, 96, 64), (32, 128, 128), (33, 129, 65), (159, 255, 100), (257, 300, 130)]
] + [("bf16", 2560, 4097, 64), ("bf16", 3071, 3072, 70), ("bf16", 2300, 4096, 2048)])
def test_store_block(fg, dtype, m, n, k, off, pad):
    from ferray_b200 import _lib as L
    r = np.random.default_rng(m * 7 + n + k)
    a, b = r.integers(-9, 10, (m, k)), r.integers(-9, 10, (k, n))
    exact = (a.astype(np.float64) @ b.astype(np.float64)).astype(np.int32)
    code = {"i8": L.FG_I8, "i16": L.FG_I16, "bf16": L.FG_BF16}[dtype]
    conv = _bf16 if dtype == "bf16" else lambda x: x.astype(dtype.replace("i", "int"))
    ct = np.float32 if dtype == "bf16" else np.int32
    da, db = fg.DeviceArray.from_numpy(conv(a)), fg.DeviceArray.from_numpy(conv(b))
    ldc = n + pad
    c0 = r.integers(-1000, 1000, off + m * ldc).astype(ct)
    ctx = fg.default_context()
    for accumulate in (0, 1):
        dc = fg.DeviceArray.from_numpy(c0)
        fg.check(ctx._lib.fg_gemm(ctx.handle, code, 0, 0, m, n, k, None, da.ptr, k, db.ptr, n, None,
                                  C.c_void_p(dc.ptr + off * 4), ldc, accumulate, None))
        ctx.sync()
        want = c0.copy()
        rows = want[off:].reshape(m, ldc)[:, :n]
        rows[:] = rows * accumulate + exact
        np.testing.assert_array_equal(dc.to_numpy(), want)
