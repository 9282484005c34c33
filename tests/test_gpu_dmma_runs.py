"""Plain DGEMM on the FP64 tensor path: 64 x 64 and 128 x 64 tiles, accumulation
runs folded in a CTA or combined by a second pass, 16-byte and 8-byte copies
(padded rows, operands off a 16-byte boundary), ragged edges, alpha and beta, and
the real-embedded ZGEMM.  Bound: (K + 4) 2^-53 ||A|| ||B||, plus the rounding
where beta reads C."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U64 = 2.0 ** -53


@pytest.mark.parametrize("pad,off", [(0, 0), (2, 2), (1, 0), (2, 1)])
@pytest.mark.parametrize("cplx,m,n,k", [
    (False, 768, 768, 768), (False, 300, 700, 2000), (False, 257, 449, 1025), (False, 1201, 333, 999),
    (False, 129, 2049, 515), (False, 10, 9, 8), (False, 100, 100, 100), (False, 500, 120, 900), (False, 1000, 1000, 1000), (False, 1537, 1536, 130), (True, 300, 251, 333),
    (True, 129, 65, 1030)])
def test_dmma_runs(fg, oracle, cplx, m, n, k, pad, off):
    from ferray_b200 import _lib as L
    r = np.random.default_rng(m + n + k + pad)
    w = 2 if cplx else 1

    def flat(rows, cols):
        x = r.standard_normal(off + rows * (cols + pad))
        return x + 1j * r.standard_normal(x.shape) if cplx else x

    def view(x, rows, cols):
        return np.ascontiguousarray(x[off:].reshape(rows, cols + pad)[:, :cols])

    fa, fb, fc = flat(m, k), flat(k, n), flat(m, n)
    da, db = fg.DeviceArray.from_numpy(fa), fg.DeviceArray.from_numpy(fb)
    a, b, c0 = view(fa, m, k), view(fb, k, n), view(fc, m, n)
    rows, cols = np.unique(np.r_[0, m - 1, r.integers(0, m, 60)]), np.unique(np.r_[0, n - 1, r.integers(0, n, 60)])
    exact = oracle.dd_sampled(a, b, rows, cols)
    scale = np.linalg.norm(a[rows]) * np.linalg.norm(b[:, cols])
    ctx = fg.default_context()
    for al, be in ((1.0, 0.0), (0.5, -2.0)):
        dc = fg.DeviceArray.from_numpy(fc)
        p = lambda d: C.c_void_p(d.ptr + 8 * w * off)  # noqa: E731
        fg.check(ctx._lib.fg_gemm(ctx.handle, L.FG_C64 if cplx else L.FG_F64, 0, 0, m, n, k, (C.c_double * 2)(al, 0.0),
                                  p(da), k + pad, p(db), n + pad, (C.c_double * 2)(be, 0.0), p(dc), n + pad, 0, None))
        ctx.sync()
        out = dc.to_numpy()
        got = view(out, m, n)[np.ix_(rows, cols)]
        ref = al * exact + be * c0[np.ix_(rows, cols)]
        assert np.linalg.norm(got - ref) <= (w * k + 4) * U64 * scale + 4 * U64 * np.linalg.norm(ref)
        if pad:
            np.testing.assert_array_equal(out[off:].reshape(m, n + pad)[:, n:], fc[off:].reshape(m, n + pad)[:, n:])


@pytest.mark.parametrize("m,n,k,count", [(32, 32, 32, 200), (55, 138, 22, 70), (65, 64, 129, 9), (250, 250, 250, 5)])
def test_dmma_stacks(fg, oracle, m, n, k, count):
    """Stacks with even and odd strides (16-byte and 8-byte copies)."""
    r = np.random.default_rng(m + n + k)
    for gap in (0, 1):
        fa, fb = r.standard_normal(count * (m * k + gap)), r.standard_normal(count * (k * n + gap))
        da, db = fg.DeviceArray.from_numpy(fa), fg.DeviceArray.from_numpy(fb)
        dc = fg.DeviceArray((count, m, n), np.float64)
        fg.gemm_batched_strided(np.float64, count, m, n, k, da, m * k + gap, db, k * n + gap, dc, m * n)
        out = dc.to_numpy()
        for i in (0, 1, count // 2, count - 1):
            a = fa.reshape(count, -1)[i, :m * k].reshape(m, k)
            b = fb.reshape(count, -1)[i, :k * n].reshape(k, n)
            err = np.linalg.norm(out[i] - oracle.dd_full(np.ascontiguousarray(a), np.ascontiguousarray(b)))
            assert err <= (k + 4) * U64 * np.linalg.norm(a) * np.linalg.norm(b)
