"""Which split SGEMM of up to 64 rows runs on the kernel that cuts B itself (slices of
A, product, combine) and which by the general path (slices of A, of B, product,
combine), and that the product is right either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,n,k,rows", [
    (1, 33, 30000, False), (64, 1, 12000, False), (33, 129, 12000, False), (16, 7, 65536, False),
    (1, 33, 16384, True), (64, 1, 8192, True), (64, 32, 30000, True), (16, 257, 30000, True)])
def test_route(fg, m, n, k, rows):
    r = np.random.default_rng(m + n + k)
    a, b = r.standard_normal((m, k), dtype=np.float32), r.standard_normal((k, n), dtype=np.float32)
    da, db, dc = fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b), fg.DeviceArray((m, n), np.float32)
    before = fg.launch_count()
    assert fg.gemm_f32(m, n, k, 1.0, da, db, 0.0, dc, mode="split")
    assert fg.launch_count() - before == (3 if rows else 4)
    exact = a.astype(np.float64) @ b.astype(np.float64)
    # two slices keep 2^-16 of a product, with random signs; the chunk sums are FP32
    bound = 8 * 2.0 ** -16 * np.sqrt(k) + 2.0 ** -24 * k
    assert np.abs(dc.to_numpy() - exact).max() <= bound
