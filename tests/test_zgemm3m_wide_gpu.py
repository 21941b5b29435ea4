"""GPU test of the one-launch zgemm3m (csrc/gemm3m.cu) with more columns than 65535
tiles of 32: products of few rows and millions of columns."""
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m,k", [(3, 2), (33, 1)])
def test_more_columns_than_one_grid_dimension(cuda, m, k):
    import torch

    n = 65535 * 32 + 1
    g = torch.Generator(device=cuda).manual_seed(m)
    rnd = lambda cnt: torch.view_as_complex(  # noqa: E731
        torch.rand(cnt, 2, dtype=torch.float64, device=cuda, generator=g) * 2 - 1)
    a, b, c = rnd(m * k), rnd(k * n), torch.zeros(m * n, dtype=torch.complex128, device=cuda)
    torch.cuda.synchronize()
    blas.zgemm3m_device("N", "N", m, n, k, 1.0, a, m, b, k, 0.0, c, m)
    torch.cuda.synchronize()
    prod = b.view(n, k) @ a.view(k, m)  # [column][row]
    # k complex products and the three-product form: sums of at most 6 k terms below 2
    assert float((c.view(n, m) - prod).abs().max()) <= 6 * k * 2 * (k + 4) * 2.0 ** -53
