"""Plain SGEMM of matrices whose tile count passes an extent of the launch grid
(65535 in y and z).  Each output is one FMA chain with k ascending, so the bits
are those of the register-staged kernel (128-row tiles, columns in x) at one
split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _f32(r, *shape):
    return r.standard_normal(shape, dtype=np.float32)


@pytest.mark.parametrize("m,n,k", [(20, 64 * 65536 + 1, 4), (64 * 65536 + 1, 2, 5)])
def test_stack_of_more_tiles_than_a_grid_extent(fg, m, n, k):
    batch = 2
    r = np.random.default_rng(m + n)
    da, db = fg.DeviceArray.from_numpy(_f32(r, batch, m, k)), fg.DeviceArray.from_numpy(_f32(r, batch, k, n))
    got = fg.matmul(da, db).to_numpy()
    with fg.tune_forced("f32", 0, 1):
        want = fg.matmul(da, db).to_numpy()
    np.testing.assert_array_equal(got, want)
