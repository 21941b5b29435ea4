"""GPU tests of the DTRSM leaf kernel and the batched inversion (csrc/trsm.cu):
orders around the 128-row blocks and the 512-row leaf, right-hand-side counts
around the 8 / 16 / 32 strips, all variants, against a solve in extended
precision on the host; the bar is the residual ||T X - alpha B|| <= n u ||T|| ||X||."""
import numpy as np
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu
U = 2.0 ** -53


@pytest.mark.parametrize("side,uplo,trans,diag", [(s, u, t, d) for s in "LR" for u in "UL"
                                                  for t in "NT" for d in "NU"])
@pytest.mark.parametrize("na,nrhs", [(1, 1), (16, 7), (127, 8), (128, 9), (129, 33), (511, 17),
                                     (513, 40), (700, 1185), (300, 2400)])
def test_leaf_edges(cuda, side, uplo, trans, diag, na, nrhs):
    import torch

    rng = np.random.default_rng(na * 31 + nrhs)
    a = rng.uniform(-1, 1, (na + 1, na))
    if diag == "U":
        a /= na
    else:
        a[np.arange(na), np.arange(na)] = na + rng.uniform(0, 1, na)
    # the other triangle and the padding row are not referenced
    keep = np.triu(np.ones((na, na)), 0) if uplo == "U" else np.tril(np.ones((na, na)), 0)
    stored = a.copy()
    stored[:na][keep == 0] = np.nan
    stored[na] = np.nan
    if diag == "U":
        stored[np.arange(na), np.arange(na)] = np.nan
    m, n = (na, nrhs) if side == "L" else (nrhs, na)
    b = rng.uniform(-1, 1, (m + 2, n))
    T = np.where(keep > 0, a[:na], 0.0)
    if diag == "U":
        np.fill_diagonal(T, 1.0)
    if trans == "T":
        T = T.T
    da = torch.from_numpy(np.ascontiguousarray(stored.T)).to(cuda)
    db = torch.from_numpy(np.ascontiguousarray(b.T)).to(cuda)
    torch.cuda.synchronize()
    blas.dtrsm_device(side, uplo, trans, diag, m, n, 0.75, da, na + 1, db, m + 2)
    torch.cuda.synchronize()
    x = db.cpu().numpy().T
    assert np.array_equal(x[m:], b[m:]), "padding rows of B were written"
    x = x[:m]
    assert np.isfinite(x).all()
    r = (T @ x if side == "L" else x @ T) - 0.75 * b[:m]
    assert np.linalg.norm(r) <= na * U * np.linalg.norm(T) * np.linalg.norm(x), np.linalg.norm(r)
