"""Ozaki scheme II at the edges of its passes: every number of moduli (each has
its own reconstruction), columns around the four a thread rebuilds and the 16 of
a residue row, imaginary columns off a 4-byte boundary, rows around the 8 of a
block, tiles on one CTA and on CTA pairs, C and operands that do not start on 16
bytes, inner shifts beyond 2^1000.  Bound as for the integer operands of P bits:
K 2^(4 - P) + K 2^-53 of ||A|| ||B||, plus the rounding where beta reads C."""
import ctypes as C

import numpy as np
import pytest

from test_gpu_ozaki2 import U64, precision_bits

pytestmark = pytest.mark.gpu


def _gemm(fg, code, moduli, m, n, k, al, a, lda, b, ldb, be, c, ldc, off):
    from ferray_b200 import _lib as L
    ctx = fg.default_context()
    w = 2 if code == L.FG_C64 else 1
    da, db, dc = (fg.DeviceArray.from_numpy(x) for x in (a, b, c))
    al, be = (C.c_double * 2)(al, 0.0), (C.c_double * 2)(be, 0.0)
    p = lambda d: C.c_void_p(d.ptr + 8 * w * off)  # noqa: E731
    fg.check(ctx._lib.fg_gemm(ctx.handle, code, L.FG_MODE_SPLIT, moduli, m, n, k, al, p(da), lda, p(db), ldb, be, p(dc),
                              ldc, 0, None))
    ctx.sync()
    return dc.to_numpy()


@pytest.mark.parametrize("cplx", [False, True])
@pytest.mark.parametrize("moduli,m,n,k,pad,off", [
    (12, 1, 1, 1, 0, 0), (13, 9, 5, 127, 1, 0), (14, 8, 15, 129, 1, 1), (15, 130, 18, 64, 2, 0), (16, 129, 257, 200, 0, 1),
    (16, 300, 131, 1300, 1, 0), (16, 513, 64, 1030, 2, 0), (17, 33, 127, 260, 3, 1), (18, 7, 34, 50, 0, 0),
    (19, 140, 63, 300, 2, 0), (20, 17, 130, 128, 1, 1)])
def test_edges(fg, oracle, cplx, moduli, m, n, k, pad, off):
    from ferray_b200 import _lib as L
    r = np.random.default_rng(moduli * 1000 + m + n + k)
    dt = np.complex128 if cplx else np.float64

    def flat(rows, cols):
        x = r.uniform(-1, 1, off + rows * (cols + pad))
        return (x + 1j * r.uniform(-1, 1, x.shape)).astype(dt) if cplx else x

    def view(x, rows, cols):
        return np.ascontiguousarray(x[off:].reshape(rows, cols + pad)[:, :cols])

    a, b, c0 = flat(m, k), flat(k, n), flat(m, n)
    code = L.FG_C64 if cplx else L.FG_F64
    exact = oracle.dd_full(view(a, m, k), view(b, k, n))
    scale = np.linalg.norm(view(a, m, k)) * np.linalg.norm(view(b, k, n))
    kw = 2 * k if cplx else k
    tol = kw * (U64 + 2.0 ** (4 - precision_bits(moduli, kw)))
    for al, be in ((1.0, 0.0), (0.5, -2.0)):
        out = _gemm(fg, code, moduli, m, n, k, al, a, k + pad, b, n + pad, be, c0, n + pad, off)
        ref = al * exact + be * view(c0, m, n)
        assert np.linalg.norm(view(out, m, n) - ref) <= tol * scale + 4 * U64 * np.linalg.norm(ref)
        keep = c0.copy()
        keep[off:].reshape(m, n + pad)[:, :n] = out[off:].reshape(m, n + pad)[:, :n]
        np.testing.assert_array_equal(out, keep)


def test_shifts_beyond_1000(fg):
    """Column k of A and row k of B 2^2040 apart: powers of two, so the scaled
    product has the bits of the plain one."""
    m, n, k = 40, 50, 30
    r = np.random.default_rng(3)
    a, b = r.integers(1, 1000, (m, k)).astype(np.float64), r.integers(1, 1000, (k, n)).astype(np.float64)
    e = np.where(np.arange(k) % 2 == 0, 1010, -1010)
    want = a @ b
    a2, b2 = np.ldexp(a, e[None, :]), np.ldexp(b, -e[:, None])
    c = np.zeros((m, n))
    assert fg.gemm_f64(m, n, k, 1.0, a2, b2, 0.0, c, mode="split", ozaki_slices=16)
    np.testing.assert_array_equal(c, want)
