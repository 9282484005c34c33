"""The few-row split SGEMM with several column tiles and K ranges a CTA: rings,
accumulators and look-ahead carried from one unit into the next, with B by TMA and as
granules.  One operand holds integers of 11 bits (two bf16 slices), the other -1, 0
and 1 (one slice), so every product and every sum (below 2^24) is exact and a missing
correction product shows at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (m, n, k, split): 297 column tiles; 161 tiles of 8 or 11 K ranges on 148 SMs
SHAPES = [(20, 37893, 200, False), (20, 37892, 200, False), (64, 37890, 70, False), (16, 20481, 3000, True),
          (16, 20484, 3000, True), (3, 20482, 4100, True), (64, 20500, 3000, True)]


@pytest.mark.parametrize("wide_a", [True, False])
@pytest.mark.parametrize("m,n,k,split", SHAPES)
def test_units(fg, m, n, k, split, wide_a):
    r = np.random.default_rng(m + n + k)
    wide = lambda *s: r.integers(-2047, 2048, s).astype(np.float32)  # noqa: E731
    unit = lambda *s: r.integers(-1, 2, s).astype(np.float32)  # noqa: E731
    a, b = (wide if wide_a else unit)(m, k), (unit if wide_a else wide)(k, n)
    da, db = fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b)
    dc = fg.DeviceArray.from_numpy(np.full((m, n), np.nan, np.float32))
    before = fg.launch_count()
    assert fg.gemm_f32(m, n, k, 1.0, da, db, 0.0, dc, mode="split")
    assert fg.launch_count() - before == 2 + split  # slices of A, product, combine
    np.testing.assert_array_equal(dc.to_numpy(), a @ b)  # exact in FP32 in any order
