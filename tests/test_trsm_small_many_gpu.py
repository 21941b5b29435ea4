"""GPU tests of small triangles against many right-hand sides (csrc/trsm.cu,
small_solve): orders around its limit of 64, alone and behind a leaf of 512, right-hand
sides around its limit of 16 per SM, all variants; residual ||T X - alpha B|| <= n u ||T|| ||X||."""
import numpy as np
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("side,uplo,trans,diag", [(s, u, t, d) for s in "LR" for u in "UL"
                                                  for t in "NT" for d in "NU"])
@pytest.mark.parametrize("na,nrhs", [(1, 9601), (17, 2368), (17, 2369), (64, 2400), (65, 2400),
                                     (512 + 33, 2500)])
def test_small_triangle_many_right_hand_sides(cuda, side, uplo, trans, diag, na, nrhs):
    import torch

    g = torch.Generator(device=cuda).manual_seed(na + nrhs)
    rand = lambda *s: torch.rand(*s, dtype=torch.float64, device=cuda, generator=g) * 2 - 1  # noqa: E731
    a = rand(na, na + 1)  # [column][row], one padding row
    if diag == "U":
        a /= na
    else:
        a.diagonal().copy_(na + a.diagonal().abs())
    A = a[:, :na].t()
    T = torch.triu(A) if uplo == "U" else torch.tril(A)
    T = T.clone()
    if diag == "U":
        T.fill_diagonal_(1.0)
    stored = torch.where(torch.triu(torch.ones_like(T)) > 0 if uplo == "U"
                         else torch.tril(torch.ones_like(T)) > 0, A, float("nan"))
    if diag == "U":
        stored.fill_diagonal_(float("nan"))  # not referenced
    a[:, :na] = stored.t()
    if trans == "T":
        T = T.t()
    m, n = (na, nrhs) if side == "L" else (nrhs, na)
    b = rand(n, m + 2)
    x = b.clone()
    torch.cuda.synchronize()
    blas.dtrsm_device(side, uplo, trans, diag, m, n, 0.75, a, na + 1, x, m + 2)
    torch.cuda.synchronize()
    assert torch.equal(x[:, m:], b[:, m:]), "padding rows of B were written"
    X, B = x[:, :m].t(), b[:, :m].t()
    r = (T @ X if side == "L" else X @ T) - 0.75 * B
    assert float(r.norm()) <= na * U * float(T.norm() * X.norm())
