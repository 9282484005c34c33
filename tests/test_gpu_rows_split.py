"""Split SGEMM of up to 64 rows (B cut into slices inside the product kernel):
row counts around the 16 / 32 / 64 row forms, column tiles of 128, K blocks of
64, K ranges, B rows at every float of a 16-byte granule, padded C, alpha and
beta.  Bound: the 3xBF16 form's 2^-15 + K 2^-24, plus the rounding of the f32
result where beta reads C."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24


def _run(fg, m, n, k, al, da, db, off, ldb, be, dc, ldc):
    from ferray_b200 import _lib as L
    ctx = fg.default_context()
    one = lambda v: C.byref(C.c_float(v))  # noqa: E731
    fg.check(ctx._lib.fg_gemm(ctx.handle, L.FG_F32, L.FG_MODE_SPLIT, 0, m, n, k, one(al), da.ptr, k, db.ptr + 4 * off,
                              ldb, one(be), dc.ptr, ldc, 0, None))
    ctx.sync()


@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (16, 128, 64), (17, 127, 63), (32, 129, 65), (33, 640, 300),
                                   (64, 257, 1025), (5, 2000, 4100)])
@pytest.mark.parametrize("pad,off", [(0, 0), (4, 0), (3, 1), (4, 2), (1, 3)])
def test_rows(fg, oracle, m, n, k, pad, off):
    r = np.random.default_rng(m + n + k + pad)
    ldb = (n + 3) // 4 * 4 + pad
    a = r.standard_normal((m, k)).astype(np.float32)
    flat = r.standard_normal(k * ldb + 8).astype(np.float32)
    b = np.ascontiguousarray(flat[off:off + k * ldb].reshape(k, ldb)[:, :n])
    c0 = r.standard_normal((m, n + 3)).astype(np.float32)
    da, db = fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(flat)
    exact = oracle.dd_full(a, b)
    scale = np.linalg.norm(a.astype(np.float64)) * np.linalg.norm(b.astype(np.float64))
    tol = 2.0 ** -15 + k * U32
    dc = fg.DeviceArray.from_numpy(c0)
    _run(fg, m, n, k, 1.0, da, db, off, ldb, 0.0, dc, n + 3)
    c = dc.to_numpy()
    np.testing.assert_array_equal(c[:, n:], c0[:, n:])
    assert np.linalg.norm(c[:, :n] - exact) <= tol * scale
    dc = fg.DeviceArray.from_numpy(c0)
    _run(fg, m, n, k, 0.5, da, db, off, ldb, -2.0, dc, n + 3)
    c = dc.to_numpy()
    ref = 0.5 * exact - 2.0 * c0[:, :n].astype(np.float64)
    np.testing.assert_array_equal(c[:, n:], c0[:, n:])
    assert np.linalg.norm(c[:, :n] - ref) <= (tol + 4 * U32) * scale + 2 * U32 * np.linalg.norm(ref)


def test_non_finite_rows_and_columns(fg):
    """Inf and NaN stay in their row (of A) or column (of B)."""
    m, n, k = 20, 300, 200
    r = np.random.default_rng(1)
    a = r.standard_normal((m, k)).astype(np.float32)
    b = r.standard_normal((k, n)).astype(np.float32)
    a[3, 5], b[7, 100], b[9, 200] = np.inf, np.nan, -np.inf
    c = np.zeros((m, n), np.float32)
    assert fg.gemm_f32(m, n, k, 1.0, a, b, 0.0, c, mode="split")
    bad = np.zeros((m, n), bool)
    bad[3], bad[:, 100], bad[:, 200] = True, True, True
    np.testing.assert_array_equal(~np.isfinite(c), bad)


@pytest.mark.parametrize("dt", [np.float32, np.float64, np.int32])
@pytest.mark.parametrize("n", [64, 66, 67])
def test_split_k_combine_widths(fg, oracle, dt, n):
    """The combine pass with 16-byte and single accesses, 16 partials, C read."""
    m, k = 33, 2100
    r = np.random.default_rng(n)
    if dt == np.int32:
        a = r.integers(-128, 128, (m, k), dtype=np.int8)
        b = r.integers(-128, 128, (k, n), dtype=np.int8)
        c0 = r.integers(-2 ** 31, 2 ** 31, (m, n), dtype=np.int64).astype(np.int32)
        c = c0.copy()
        with fg.tune_forced("i8", 1, 16):
            assert fg.gemm_i8_signed(m, n, k, a, b, c, accumulate=True)
        np.testing.assert_array_equal(c, oracle.gemm_i8_signed(a, b, c=c0, accumulate=True))
        return
    a, b = r.uniform(-1, 1, (m, k)).astype(dt), r.uniform(-1, 1, (k, n)).astype(dt)
    c0 = r.uniform(-1, 1, (m, n)).astype(dt)
    c = c0.copy()
    gemm, op, u = (fg.gemm_f32, "f32", U32) if dt == np.float32 else (fg.gemm_f64, "f64", 2.0 ** -53)
    with fg.tune_forced(op, 1, 16):
        assert gemm(m, n, k, 0.5, a, b, 2.0, c)
    ref = 0.5 * oracle.dd_full(a, b) + 2.0 * c0.astype(np.float64)
    scale = np.linalg.norm(a.astype(np.float64)) * np.linalg.norm(b.astype(np.float64))
    assert np.linalg.norm(c - ref) <= (k + 4) * u * scale + 2 * u * np.linalg.norm(ref)
