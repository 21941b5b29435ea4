"""GPU tests of the length of the FP64 GEMM's chains of additions (csrc/dgemm_fp64.cu):
the error of a product of uniform random matrices against extended precision.

A chain of c additions of terms of one size has a squared error of c (c + 1) / 2 terms
of (r u)^2, r the root mean square rounding error in units of u = 2^-53 (0.44, measured
on chains of 128 to 2048; 1/sqrt(3) times the mean mantissa); S chains added in turn
S (S + 1) / 2 terms of c (r u)^2 more; relative to the K = c S terms of the result that
is r u sqrt((c + 1) / 2 + (S + 1) / 2).  The bar allows 1.25 times it."""
import numpy as np
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu


# chain: what 64x64 tiles in slices of K give (at most 8 slices and 1024 tiles x slices)
@pytest.mark.parametrize("m,n,k,chain", [
    (64, 64, 128, 16), (96, 200, 256, 32), (200, 170, 1600, 208), (512, 512, 512, 64),
    (640, 640, 1024, 128), (1024, 1024, 1024, 256), (128, 2048, 128, 16), (300, 65, 2000, 256)])
@pytest.mark.parametrize("ta,tb,pad", [("N", "N", 0), ("T", "N", 1), ("N", "T", 0)])
def test_chains_are_no_longer_than_a_slice(cuda, m, n, k, chain, ta, tb, pad):
    import torch

    rng = np.random.default_rng(m + n + k)
    a, b = rng.uniform(-1, 1, (m, k)), rng.uniform(-1, 1, (k, n))

    def operand(x, t):  # column-major, padded
        x = x if t == "N" else x.T
        buf = np.zeros((x.shape[1], x.shape[0] + pad))
        buf[:, :x.shape[0]] = x.T
        return torch.from_numpy(buf).to(cuda), buf.shape[1]

    (da, lda), (db, ldb) = operand(a, ta), operand(b, tb)
    dc = torch.zeros((n, m), dtype=torch.float64, device=cuda)
    torch.cuda.synchronize()
    blas.dgemm_device(ta, tb, m, n, k, 1.0, da, lda, db, ldb, 0.0, dc, m, method="fp64")
    torch.cuda.synchronize()
    rows = slice(0, min(m, 128))  # enough for a norm
    ref = a[rows].astype(np.longdouble) @ b[:, :64].astype(np.longdouble)
    got = dc.cpu().numpy().T[rows, :64]
    err = float(np.sqrt(((got - ref) ** 2).sum() / (ref ** 2).sum()))
    chains = -(-k // chain)
    assert err <= 1.25 * 0.44 * 2.0 ** -53 * np.sqrt((chain + 1) / 2 + (chains + 1) / 2), err
