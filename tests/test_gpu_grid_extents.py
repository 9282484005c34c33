"""Plain SGEMM of matrices whose tile count passes an extent of the launch grid
(65535 in y and z).  Each output is one FMA chain with k ascending, so the bits
are those of the register-staged kernel (128-row tiles, columns in x) at one
split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _f32(r, *shape):
    return r.standard_normal(shape, dtype=np.float32)


@pytest.mark.parametrize("m,n,k", [(32, 64 * 65536 + 1, 16), (64 * 65536 + 1, 2, 5)])
def test_stack_of_more_tiles_than_a_grid_extent(fg, m, n, k):
    batch = 2
    r = np.random.default_rng(m + n)
    da, db = fg.DeviceArray.from_numpy(_f32(r, batch, m, k)), fg.DeviceArray.from_numpy(_f32(r, batch, k, n))
    got = fg.matmul(da, db).to_numpy()
    with fg.tune_forced("f32", 0, 1):
        want = fg.matmul(da, db).to_numpy()
    np.testing.assert_array_equal(got, want)


def _sampled_rows(m):
    return np.unique(np.r_[0:3, 16 * 65535 - 2:16 * 65535 + 3, 64 * 65535 - 2:64 * 65535 + 3, m // 2, m - 3:m]).clip(max=m - 1)


@pytest.mark.parametrize("cplx,m,n,k", [(False, 16 * 65535 + 1, 160, 144), (True, 64 * 65535 + 1, 65, 65)])
def test_more_rows_than_low_tiles_allow(fg, cplx, m, n, k):
    """Beyond 65535 tiles of 16 (64) rows a product stays on the packed kernel (for
    complex operands the real embedding on it), with a tile that fits: the transpose
    of A and one product, after the embedding of B."""
    import torch
    from ferray_b200 import _lib as L
    gen = torch.Generator(device="cuda").manual_seed(m)
    t = torch.complex64 if cplx else torch.float32
    a, b = (torch.randn(s, generator=gen, device="cuda", dtype=t) for s in ((m, k), (k, n)))
    c = torch.full((m, n), float("nan"), device="cuda", dtype=t)
    assert fg.tune_lookup("f32", m, (1 + cplx) * n, (1 + cplx) * k) == (4, 1)
    one, zero = np.array([1, 0], np.float32), np.zeros(2, np.float32)
    ctx = fg.default_context()

    def gemm(rows, x, out):
        torch.cuda.synchronize()
        before = fg.launch_count()
        fg.check(ctx._lib.fg_gemm(ctx.handle, L.FG_C32 if cplx else L.FG_F32, 0, 0, rows, n, k, one.ctypes.data,
                                  x.data_ptr(), k, b.data_ptr(), n, zero.ctypes.data, out.data_ptr(), n, 0, None))
        ctx.sync()
        return fg.launch_count() - before

    assert gemm(m, a, c) == 2 + cplx
    rows = torch.from_numpy(np.unique(_sampled_rows(m))).cuda()
    # the same rows alone, 128 of them: one split, so the same chain of k
    few = a[rows].repeat(128 // len(rows) + 1, 1)[:128].contiguous()
    want = torch.empty((128, n), device="cuda", dtype=t)
    with fg.tune_forced("f32", 4, 1):
        gemm(128, few, want)
    torch.testing.assert_close(c[rows], want[:len(rows)], rtol=0, atol=0)
    exact = few[:len(rows)].to(torch.complex128) @ b.to(torch.complex128)
    bound = (2 if cplx else 1) * k * 2.0 ** -24 * (few[:len(rows)].abs().double() @ b.abs().double())
    assert ((c[rows] - exact).abs() <= 2 * bound).all()
