"""GPU tests of the length of the chains of additions in a DTRSM leaf
(csrc/trsm.cu, trsm_leaf_kernel).

A unit triangle with one row off the identity has an inverse that is known exactly, and
the solution's row is a product of length 128 with random right-hand sides.  A chain of c
additions has a relative error of r u sqrt((c + 1) / 2), r = 0.44 measured on DMMA
chains, S of them added in turn sqrt((S + 1) / 2) more in squares; the bar is 1.25 times
that of chains of 16."""
import numpy as np
import pytest

from gemm_avx512f_b200 import blas

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nrhs", [1000, 2000, 4000])  # strips of 8, 16 and 32
@pytest.mark.parametrize("row,first", [(127, 0), (255, 0)])  # the inverse's product; an update
def test_chains_of_a_leaf(cuda, nrhs, row, first):
    import torch

    n, length = 256, 128 if row == 255 else 127
    rng = np.random.default_rng(nrhs + row)
    T = np.eye(n)
    u = rng.uniform(-1, 1, length)
    T[row, first:first + length] = u
    b = rng.uniform(-1, 1, (n, nrhs))
    b[row] = 0.0  # nothing else in the row's sum
    a = torch.from_numpy(np.ascontiguousarray(T.T)).to(cuda)
    x = torch.from_numpy(np.ascontiguousarray(b.T)).to(cuda)
    torch.cuda.synchronize()
    blas.dtrsm_device("L", "L", "N", "U", n, nrhs, 1.0, a, n, x, n)
    torch.cuda.synchronize()
    got = x.cpu().numpy().T
    keep = np.arange(n) != row
    assert np.array_equal(got[keep], b[keep])
    ref = -(u.astype(np.longdouble) @ b[first:first + length].astype(np.longdouble))
    err = float(np.sqrt(((got[row] - ref) ** 2).sum() / (ref ** 2).sum()))
    c, chains = 16, 8
    assert err <= 1.25 * 0.44 * 2.0 ** -53 * np.sqrt((c + 1) / 2 + (chains + 1) / 2), err
