"""Split CGEMM as the real GEMM (M x 2K) (2K x 2N) of the interleaved operands
on every tile variant and split-K count, at sizes around the tile, chunk and
16-byte-group edges, with beta read from C.

Bound: the embedded product has inner dimension 2K and each complex entry of C
is two of its entries, so the real split bound 2^-15 + 2K 2^-24 (3xBF16;
2^-21 + 2K 2^-24 for the FP16 slices, 2K 2^-24 + 2^-23 for 6xBF16) holds
normwise on C; beta adds the rounding of the f32 result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

U32 = 2.0 ** -24
REP = {("split", 2): 2.0 ** -15, ("split", 3): 2.0 ** -23, ("split_f16", 0): 2.0 ** -21}


@pytest.mark.parametrize("variant,splits", [(0, 1), (1, 3), (2, 1), (2, 2)])
@pytest.mark.parametrize("m,n,k", [(1, 1, 1), (3, 5, 33), (129, 63, 65), (256, 66, 128), (70, 131, 515)])
@pytest.mark.parametrize("mode,slices", list(REP))
def test_split_cgemm_embedding(fg, oracle, variant, splits, m, n, k, mode, slices):
    r = np.random.default_rng(m * 7 + n + k)
    cplx = lambda *s: (r.standard_normal(s) + 1j * r.standard_normal(s)).astype(np.complex64)  # noqa: E731
    a, b, c0 = cplx(m, k), cplx(k, n), cplx(m, n)
    exact = oracle.dd_full(a.astype(np.complex128), b.astype(np.complex128))
    scale = np.linalg.norm(a.astype(np.complex128)) * np.linalg.norm(b.astype(np.complex128))
    tol = REP[(mode, slices)] + 2 * k * U32
    with fg.tune_forced("split_f32", variant, splits):
        c = np.zeros((m, n), np.complex64)
        assert fg.gemm_c32(m, n, k, 1.0, 0.0, a, b, 0.0, 0.0, c, mode=mode, bf16_slices=slices)
        assert np.linalg.norm(c - exact) <= tol * scale
        c = c0.copy()
        assert fg.gemm_c32(m, n, k, 0.5, 0.0, a, b, -2.0, 0.0, c, mode=mode, bf16_slices=slices)
    ref = 0.5 * exact - 2.0 * c0.astype(np.complex128)
    assert np.linalg.norm(c - ref) <= (tol + 4 * U32) * scale + 2 * U32 * np.linalg.norm(ref)
