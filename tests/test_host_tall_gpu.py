"""GPU test of pageable host operands with few long columns (csrc/api.cu): a bounce
chunk holds one column or a few, whose copies several threads share."""
import numpy as np
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("m,n,k,pad", [(1100003, 3, 2, 0), (1100003, 3, 2, 5), (600001, 2, 3, 1),
                                       (130000, 9, 5, 3), (2500000, 1, 1, 0)])
def test_tall_operands(cuda, dtype, m, n, k, pad):
    rng = np.random.default_rng(m + pad)
    fn = blas.dgemm if dtype == np.float64 else blas.sgemm
    a = np.asfortranarray(rng.uniform(-1, 1, (m + pad, k)).astype(dtype))
    b = np.asfortranarray(rng.uniform(-1, 1, (k, n)).astype(dtype))
    c = np.asfortranarray(rng.uniform(-1, 1, (m + pad, n)).astype(dtype))
    got = c.copy(order="F")
    fn("N", "N", m, n, k, 1.5, a, m + pad, b, k, 0.5, got, m + pad)
    ref = 1.5 * (a[:m].astype(np.float64) @ b) + 0.5 * c[:m]
    u = np.finfo(dtype).eps / 2
    assert np.abs(got[:m] - ref).max() <= (k + 4) * u * (1.5 * k + 0.5)
    assert np.array_equal(got[m:], c[m:])
    # the transposed operand is the tall one: its columns are the long K
    if pad == 0:
        t = np.asfortranarray(np.zeros((k, n), dtype))
        fn("T", "N", k, n, m, 1.0, a, m, c, m, 0.0, t, k)
        reft = a[:m].astype(np.float64).T @ c[:m].astype(np.float64)
        bound = m * u * (np.abs(a[:m]).astype(np.float64).T @ np.abs(c[:m]).astype(np.float64))
        assert (np.abs(t - reft) <= bound).all()
