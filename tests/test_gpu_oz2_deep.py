"""The rebuilt product of scheme II at a long K, where |C'| reaches 2^135 and the top
digit of the four- and five-digit forms is in use: 49-bit integers, exactly held by
the scaled entries (P >= 53), so every output is the double nearest to the integer
product."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("signs", [False, True])
@pytest.mark.parametrize("moduli", [16, 17, 18, 19, 20])
def test_deep(fg, moduli, signs):
    r = np.random.default_rng(moduli)
    m, n, k = 6, 5, 100000
    a, b = r.integers(2 ** 48, 2 ** 49, (m, k)), r.integers(2 ** 48, 2 ** 49, (k, n))
    if signs:
        a *= r.choice([-1, 1], (m, k))
    c = np.zeros((m, n))
    assert fg.gemm_f64(m, n, k, 1.0, a.astype(np.float64), b.astype(np.float64), 0.0, c, mode="split",
                       ozaki_slices=moduli)
    ai, bi = a.tolist(), b.T.tolist()
    want = [[float(sum(x * y for x, y in zip(row, col))) for col in bi] for row in ai]
    np.testing.assert_array_equal(c, want)
