"""Stacked and ragged plain SGEMM on 64 x 64 tiles of 64 threads: the four
half-tile loops, K tails, both load widths, alpha / beta and broadcast strides.
Each output is one FMA chain with k ascending, so the bits are those of the
register-staged kernel at one split."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EDGES = [1, 31, 32, 33, 64, 65, 96, 97]


def _reference(fg, a, b):
    """One product by the register-staged kernel at one split, as a stack of two
    (a lone row or column would go to the matrix-vector kernels)."""
    with fg.tune_forced("f32", 0, 1):
        return fg.matmul(np.stack([a, a]), np.stack([b, b]))[0]


@pytest.mark.parametrize("k", [1, 7, 8, 16, 17, 40])
@pytest.mark.parametrize("m,n", [(1, 1), (31, 33), (32, 64), (33, 32), (64, 97), (65, 31), (96, 80), (97, 65)])
def test_stack(fg, m, n, k):
    batch = 150  # more tiles than SMs
    r = np.random.default_rng(m * 100 + n * 10 + k)
    a = r.standard_normal((batch, m, k)).astype(np.float32)
    b = r.standard_normal((batch, k, n)).astype(np.float32)
    da, db = fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b)
    got = fg.matmul(da, db).to_numpy()
    for i in (0, 1, batch - 1):
        np.testing.assert_array_equal(got[i], _reference(fg, a[i], b[i]))
    # one B for the whole stack, alpha and beta
    c0 = r.standard_normal((batch, m, n)).astype(np.float32)
    out = []
    for forced in (False, True):
        dc = fg.DeviceArray.from_numpy(c0)
        run = lambda: fg.gemm_batched_strided(np.float32, batch, m, n, k, da, m * k, db, 0, dc, m * n,  # noqa: E731
                                              alpha=0.5, beta=-2.0)
        if forced:
            with fg.tune_forced("f32", 0, 1):
                run()
        else:
            run()
        out.append(dc.to_numpy())
    np.testing.assert_array_equal(out[0], out[1])


def test_ragged_edges(fg):
    r = np.random.default_rng(5)
    shapes = [(m, n, k) for m in EDGES for n in EDGES for k in (1, 15, 16, 17, 33)]
    arrays, problems = [], []
    for m, n, k in shapes:
        a = r.standard_normal((m, k)).astype(np.float32)
        b = r.standard_normal((k, n)).astype(np.float32)
        c = fg.DeviceArray.from_numpy(np.full((m, n), np.nan, np.float32))
        arrays.append((a, b, c))
        problems.append((m, n, k, fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b), c))
    fg.gemm_grouped(problems)
    for a, b, c in arrays:
        np.testing.assert_array_equal(c.to_numpy(), _reference(fg, a, b))


@pytest.mark.parametrize("m,n,k", [(23, 29, 240), (64, 64, 500), (33, 97, 1000), (70, 20, 2000)])
def test_stack_keeps_the_split_rounding(fg, m, n, k):
    """Where the table splits K, the stack kernel closes its accumulators at the
    same places and adds them in the same order: same bits as the split form."""
    batch = 160
    _, splits = fg.tune_lookup("f32", m, n, k)
    assert splits > 1
    r = np.random.default_rng(k)
    a = r.standard_normal((batch, m, k)).astype(np.float32)
    b = r.standard_normal((batch, k, n)).astype(np.float32)
    da, db = fg.DeviceArray.from_numpy(a), fg.DeviceArray.from_numpy(b)
    got = fg.matmul(da, db).to_numpy()
    with fg.tune_forced("f32", 0, splits):
        want = fg.matmul(da, db).to_numpy()
    np.testing.assert_array_equal(got, want)
