"""What the dispatch does without room for its scratch memory: another way with the
tuned accumulation runs (and so the same rounding) where there is one, else
OutOfMemory.  The room is taken away by a memory pool with a size limit."""
import contextlib

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
MB = 1 << 20


@contextlib.contextmanager
def scratch_limit(nbytes):
    """Stream-ordered allocations of device 0 come from a pool of at most nbytes."""
    from cuda.bindings import driver as cu

    def ok(r):
        assert r[0] == cu.CUresult.CUDA_SUCCESS, r[0]
        return r[1] if len(r) > 1 else None
    p = cu.CUmemPoolProps()
    p.allocType = cu.CUmemAllocationType.CU_MEM_ALLOCATION_TYPE_PINNED
    p.handleTypes = cu.CUmemAllocationHandleType.CU_MEM_HANDLE_TYPE_NONE
    p.location.type = cu.CUmemLocationType.CU_MEM_LOCATION_TYPE_DEVICE
    p.location.id = 0
    p.maxSize = nbytes
    pool = ok(cu.cuMemPoolCreate(p))
    default = ok(cu.cuDeviceGetDefaultMemPool(0))
    ok(cu.cuDeviceSetMemPool(0, pool))
    try:
        yield
    finally:
        ok(cu.cuDeviceSetMemPool(0, default))
        ok(cu.cuMemPoolDestroy(pool))


def _operands(fg, dtype, *shapes):
    r = np.random.default_rng(sum(sum(s) for s in shapes))
    return [fg.DeviceArray.from_numpy(r.standard_normal(s, dtype=np.float32) if dtype is np.float32 else
                                      (r.standard_normal(s) + 1j * r.standard_normal(s)).astype(dtype)) for s in shapes]


@pytest.mark.parametrize("m,n,k,room", [
    (2048, 2048, 2048, 32),    # A's copy fits (16 MB), two partial products (34 MB) do not: the table has one split
    (7000, 64, 10000, 64),     # 280 MB for A's copy: the register-staged kernel needs none (29 MB of partial products)
])
def test_plain_keeps_the_tuned_runs(fg, m, n, k, room):
    variant, splits = fg.tune_lookup("f32", m, n, k)
    a, b = _operands(fg, np.float32, (m, k), (k, n))
    with scratch_limit(room * MB):
        got = fg.matmul(a, b).to_numpy()
    with fg.tune_forced("f32", 0, splits):
        want = fg.matmul(a, b).to_numpy()
    np.testing.assert_array_equal(got, want)


def test_stack_without_room(fg):
    """96 MB for A's copies: one CTA of 64 threads a tile needs none."""
    batch, m, n, k = 40, 300, 700, 2000
    _, splits = fg.tune_lookup("f32", m, n, k)
    a, b = _operands(fg, np.float32, (batch, m, k), (batch, k, n))
    with scratch_limit(32 * MB):
        got = fg.matmul(a, b).to_numpy()
    with fg.tune_forced("f32", 0, splits):
        want = fg.matmul(a, b).to_numpy()
    np.testing.assert_array_equal(got, want)


def test_no_room_for_the_packed_copy(fg):
    a, b = _operands(fg, np.float32, (5000, 8000), (8000, 1000))
    assert fg.tune_lookup("f32", 5000, 1000, 8000)[0] == 4
    with scratch_limit(32 * MB), pytest.raises(fg.OutOfMemory):
        fg.matmul(a, b)


def test_split_without_room_for_the_partial_products(fg):
    """1 GB of them, 34 MB of planes: an error for a real product (one run over K
    would round differently), one run for a complex one."""
    a, b = _operands(fg, np.float32, (4096, 1024), (1024, 4096))
    with fg.tune_forced("split_f32", 2, 16), scratch_limit(512 * MB), pytest.raises(fg.OutOfMemory):
        fg.matmul(a, b, mode="split")
    a, b = _operands(fg, np.complex64, (4096, 512), (512, 2048))
    with fg.tune_forced("split_f32", 2, 16), scratch_limit(512 * MB):
        got = fg.matmul(a, b, mode="split").to_numpy()
    with fg.tune_forced("split_f32", 2, 1):
        want = fg.matmul(a, b, mode="split").to_numpy()
    np.testing.assert_array_equal(got, want)


@pytest.mark.parametrize("batch,m,n,k", [(40000, 16, 100, 1024), (33000, 16, 16, 2000)])
def test_more_splits_than_the_grid_allows(fg, batch, m, n, k):
    """A stack whose tuned splits times its matrices pass the grid's z extent keeps
    the tuned runs (the split count is also capped by 1 GiB of partial products)."""
    splits = min(fg.tune_lookup("f32", m, n, k)[1], (1 << 30) // (4 * batch * m * n))
    assert splits * batch > 65535
    a, b = _operands(fg, np.float32, (m, k), (k, n))

    def stack(count):  # the same two operands for every matrix
        c = fg.DeviceArray((count, m, n), np.float32)
        fg.gemm_batched_strided(np.float32, count, m, n, k, a, 0, b, 0, c, m * n)
        return c.to_numpy()
    got = stack(batch)
    with fg.tune_forced("f32", 0, splits):
        want = stack(2)
    np.testing.assert_array_equal(got[[0, batch // 2, batch - 1]], want[[0, 0, 0]])
