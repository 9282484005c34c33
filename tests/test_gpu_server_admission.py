"""The server's estimate of a split f64 / c64 request covers the residue-byte planes
of the product, whose rows are padded to 16 bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,n", [(np.float64, 1), (np.float64, 17), (np.complex128, 1)])
def test_split_request_counts_the_padded_planes(fg, dtype, n):
    m, k, moduli = 5000, 3, 16
    a, b, c = (fg.DeviceArray.from_numpy(np.ones(s, dtype)) for s in ((m, k), (k, n), (m, n)))
    wide = 2 if dtype is np.complex128 else 1  # columns of the real embedding
    planes = moduli * m * (-(-wide * n // 16) * 16)
    srv = fg.Server(hbm_budget_bytes=1 << 30)
    srv.wait(srv.submit(a, b, c, "split"), timeout_ms=60000)
    peak = srv.stats()["hbm_peak"]
    srv.stop()
    np.testing.assert_array_equal(c.to_numpy(), np.full((m, n), k, dtype))
    assert peak >= planes + a.nbytes + b.nbytes + c.nbytes
