"""Which plain SGEMM of one matrix leaves the table's register-staged tile for the
packed kernel (one launch more: the transpose of A), and that the product is right
either way."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STAGED = [(7000, 9, 3000), (300, 33, 3000), (1000, 64, 2000), (30000, 5, 1100), (300, 33, 6000), (220, 65, 3365),
          (279, 195, 802)]
PACKED = [(33, 7000, 1100), (3000, 64, 2000), (64, 20, 12000), (17, 1000, 3000), (220, 130, 3365)]


@pytest.mark.parametrize("m,n,k,packed", [s + (False,) for s in STAGED] + [s + (True,) for s in PACKED])
def test_route(fg, oracle, m, n, k, packed):
    variant, splits = fg.tune_lookup("f32", m, n, k)
    assert variant < 4 and splits > 1
    r = np.random.default_rng(m + n + k)
    a, b = r.uniform(-1, 1, (m, k)).astype(np.float32), r.uniform(-1, 1, (k, n)).astype(np.float32)
    da, db, dc = fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b), fg.DeviceArray((m, n), np.float32)
    before = fg.launch_count()
    assert fg.gemm_f32(m, n, k, 1.0, da, db, 0.0, dc)
    assert fg.launch_count() - before == (3 if packed else 2)  # (transpose,) product, combine
    assert oracle.error_vs_dd(a, b, dc.to_numpy()) <= k * 2.0 ** -24
