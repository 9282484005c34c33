"""The rebuilt product of scheme II is rounded once.  Entries are 49-bit integers,
exactly held by the scaled ones (P >= 55), so the emulated product is exact before
the last step: every output is the double nearest to the integer product (at most
one in 1000 its neighbour: what is rounded below the last place is 2^-40 of it)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("moduli", [16, 17, 18, 19, 20])
def test_rounded_once(fg, moduli):
    r = np.random.default_rng(moduli)
    m, n, k = 96, 88, 1
    a = r.integers(2 ** 48, 2 ** 49, (m, k)) * r.choice([-1, 1], (m, k))
    b = r.integers(2 ** 48, 2 ** 49, (k, n))
    c = np.zeros((m, n))
    assert fg.gemm_f64(m, n, k, 1.0, a.astype(np.float64), b.astype(np.float64), 0.0, c, mode="split",
                       ozaki_slices=moduli)
    want = np.array([[float(int(x) * int(y)) for y in b[0]] for x in a[:, 0]])
    assert np.mean(c != want) <= 1e-3
