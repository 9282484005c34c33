"""Plain FP32 grouped batches of few tiles, which are cut into 32 x 32 ones: sizes
around their edges and around the count (3 / 2 a SM) up to which they are, bit for bit
the register-staged kernel's result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 7, 221, 223])
def test_few_tiles(fg, count):
    sms = fg.default_context().info()["sm_count"]
    r = np.random.default_rng(count)
    shapes = [(33, 64, 17), (1, 1, 1), (64, 64, 100), (32, 33, 16), (31, 5, 300), (64, 32, 15)]
    shapes = [shapes[i % len(shapes)] for i in range(count if count < 200 else count * sms // 148)]
    arrays, problems = [], []
    for m, n, k in shapes:
        a, b = r.standard_normal((m, k), dtype=np.float32), r.standard_normal((k, n), dtype=np.float32)
        c = fg.DeviceArray.from_numpy(np.full((m, n), np.nan, np.float32))
        arrays.append((a, b, c))
        problems.append((m, n, k, fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b), c))
    fg.gemm_grouped(problems)
    for a, b, c in arrays:
        with fg.tune_forced("f32", 0, 1):
            want = fg.matmul(np.stack([a, a]), np.stack([b, b]))[0]
        np.testing.assert_array_equal(c.to_numpy(), want)


def test_few_large(fg):
    """More tiles of 32 than of 64 by four: 2 x 500 x 700 (176 whole tiles, 704 small)."""
    r = np.random.default_rng(3)
    problems, arrays = [], []
    for m, n, k in [(500, 700, 130), (470, 641, 33)]:
        a, b = r.standard_normal((m, k), dtype=np.float32), r.standard_normal((k, n), dtype=np.float32)
        c = fg.DeviceArray.from_numpy(np.full((m, n), np.nan, np.float32))
        arrays.append((a, b, c))
        problems.append((m, n, k, fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b), c))
    plan = fg.GroupedPlan(problems)
    plan.run()
    for a, b, c in arrays:
        with fg.tune_forced("f32", 0, 1):
            want = fg.matmul(np.stack([a, a]), np.stack([b, b]))[0]
        np.testing.assert_array_equal(c.to_numpy(), want)
    plan.close()
