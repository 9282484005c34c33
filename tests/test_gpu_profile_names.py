"""fg_profile_* lists a plain product under the kernel that ran, once a call."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,shape,name", [
    (np.float32, (512, 96, 80, 64), "sgemm_tile64"),       # stacks
    (np.float32, (3, 700, 700, 2000), "ffma_sgemm"),
    (np.float32, (1, 3000, 64, 2000), "ffma_sgemm"),       # the table has a register-staged tile
    (np.float32, (1, 1024, 1024, 1024), "ffma_sgemm"),
    (np.float32, (1, 300, 33, 3000), "simt_sgemm"),
    (np.float64, (1, 100, 100, 100), "dmma_dgemm"),
    (np.float64, (1, 100, 100, 8), "simt_dgemm"),
    (np.complex64, (1, 600, 600, 600), "simt_cgemm"),
    (np.complex128, (1, 300, 300, 300), "simt_zgemm"),
])
def test_profile_name(fg, dtype, shape, name):
    from ferray_b200 import _lib as L
    batch, m, n, k = shape
    a, b = (fg.DeviceArray.from_numpy(np.ones((batch,) * (batch > 1) + s, dtype)) for s in ((m, k), (k, n)))
    lib = L.load()
    ents, cnt = (L.fg_profile_entry * 16)(), C.c_int()
    lib.fg_profile_enable(1)
    try:
        fg.matmul(a, b)
    finally:
        lib.fg_profile_enable(0)
        lib.fg_profile_collect(ents, 16, C.byref(cnt))
    assert [(e.name.decode(), e.launches) for e in ents[:cnt.value]] == [(name, 1)]
