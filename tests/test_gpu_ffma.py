"""Plain SGEMM on the paired-FMA kernel: every tile and the row-shifted B form.

The kernel keeps the per-output k order of the register-staged kernel, so at an
equal split count the bits are the same whatever the tile, the alignment of B's
rows, the leading dimensions and the batch strides; shapes lie on the edges of
the tiles (16, 32, 64, 128 rows; 64, 128 columns), of the 16-deep K blocks and
of the 64-deep split units."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (16, 128, 16), (17, 129, 65), (32, 64, 130), (33, 257, 64), (64, 127, 515), (129, 65, 33),
          (128, 512, 1030), (300, 700, 200), (3, 2000, 1100)]


def _gemm(fg, dt, m, n, k, al, a, lda, b, ldb, be, c, ldc):
    ctx = fg.default_context()
    one = lambda v: C.byref(C.c_float(v))  # noqa: E731
    fg.check(ctx._lib.fg_gemm(ctx.handle, dt, 0, 0, m, n, k, one(al), a, lda, b, ldb, one(be), c, ldc, 0, None))
    ctx.sync()


@pytest.mark.parametrize("splits", [1, 2, 16])
@pytest.mark.parametrize("m,n,k", SHAPES)
def test_tiles_bit_identical_at_any_alignment(fg, m, n, k, splits):
    from ferray_b200 import _lib as L
    r = np.random.default_rng(m + 3 * n + 7 * k)
    pad_a, pad_b, pad_c = 3, 5, 2
    a = r.standard_normal((m, k + pad_a)).astype(np.float32)
    c0 = r.standard_normal((m, n + pad_c)).astype(np.float32)
    da = fg.DeviceArray.from_numpy(a)
    flat = r.standard_normal(k * (n + pad_b) + 8).astype(np.float32)
    db = fg.DeviceArray.from_numpy(flat)
    # ldb odd / a multiple of 4, base at each float of a 16-byte granule
    for ldb, off in [(n + pad_b, 0), (n + pad_b, 3), ((n + 3) // 4 * 4, 0), ((n + 3) // 4 * 4, 1), ((n + 3) // 4 * 4, 2)]:
        out = []
        for variant in (0, 4, 5):
            dc = fg.DeviceArray.from_numpy(c0)
            with fg.tune_forced("f32", variant, splits):
                _gemm(fg, L.FG_F32, m, n, k, 0.75, da.ptr, k + pad_a, db.ptr + 4 * off, ldb, -1.5, dc.ptr, n + pad_c)
            out.append(dc.to_numpy())
        np.testing.assert_array_equal(out[0], out[1])
        np.testing.assert_array_equal(out[0], out[2])
        np.testing.assert_array_equal(out[1][:, n:], c0[:, n:])  # past the row end: untouched


@pytest.mark.parametrize("m,n,k", SHAPES)
def test_default_choice_within_bound(fg, oracle, m, n, k):
    r = np.random.default_rng(m * n + k)
    a = r.uniform(-1, 1, (m, k)).astype(np.float32)
    b = r.uniform(-1, 1, (k, n)).astype(np.float32)
    c = np.full((m, n), np.nan, np.float32)
    assert fg.gemm_f32(m, n, k, 1.0, a, b, 0.0, c)
    assert oracle.error_vs_dd(a, b, c) <= k * 2.0 ** -24


@pytest.mark.parametrize("stride_b", [300 * 45, 300 * 45 + 1, 0])
def test_batch_strides(fg, stride_b):
    """B matrices whose distance breaks the 16-byte rule although one matrix keeps it."""
    batch, m, n, k = 3, 70, 44, 300
    r = np.random.default_rng(stride_b)
    a = r.standard_normal((batch, m, k)).astype(np.float32)
    b = r.standard_normal(batch * (k * n + 301)).astype(np.float32)
    da, db = fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b)
    out = []
    for variant in (0, 4):
        dc = fg.DeviceArray((batch, m, n), np.float32)
        with fg.tune_forced("f32", variant, 2):
            fg.gemm_batched_strided(np.float32, batch, m, n, k, da, m * k, db, stride_b, dc, m * n)
        out.append(dc.to_numpy())
    np.testing.assert_array_equal(out[0], out[1])
